// Plain kernels: one CUDA kernel per reference subroutine, FP64 (RP = DP) and
// FP32 (RP = SP), same argument meaning and array layout as the reference.
//
//   horizontal_flux            dyn_horiz_adv_flux/src/mod_src_tracer.f90:42-379
//   horizontal_limiter_thuburn dyn_horiz_adv_limiter/src/mod_src_tracer.f90:42-430
//   vertical_limiter_thuburn   dyn_vert_adv_limiter/src/mod_src_tracer.f90:41-243
//   COMM_data_transfer         communication/src/mod_comm.f90:1506-1891 (as a gather)
//
// This file is compiled with --fmad=false: every expression keeps the
// reference's operation order and no multiply-add is contracted, so the FP64
// results equal a non-contracting CPU build of the reference bit for bit.
//
// Thread mapping.  The reference loops over faces and scatters each face
// value to both cells (flx_h(ij,1) and flx_h(ip1j,4), Qin(ij,1) and
// Qin(ip1j,4), q_a(ij,1) and q_a(ip1j,4)).  Here one thread owns one cell
// (i,j) of one (k,l) slab, evaluates the three faces the reference attaches to
// that cell, and writes both sides; every output element has exactly one
// writer, and halo elements that no face loop reaches get the zero the
// reference writes first.  Index (i,j) is 1-based as in the reference,
// ij = (j-1)*gall_1d + i, arrays are addressed with ij-1.
#include <cuda_runtime.h>

#include <cfloat>
#include <cstdint>

#include "plain_kernels.cuh"
#include "quotients.cuh"

namespace icoadv {

template <typename T> struct Num;
template <> struct Num<double> {
  static __device__ __forceinline__ double eps() { return DBL_EPSILON; }
  static __device__ __forceinline__ double big() { return DBL_MAX; }
};
template <> struct Num<float> {
  static __device__ __forceinline__ float eps() { return FLT_EPSILON; }
  static __device__ __forceinline__ float big() { return FLT_MAX; }
};

// Fortran MIN/MAX of two values and SIGN(a,b) with IEEE signed zero.
template <typename T> __device__ __forceinline__ T mn(T a, T b) { return (b < a) ? b : a; }
template <typename T> __device__ __forceinline__ T mx(T a, T b) { return (b > a) ? b : a; }
template <typename T> __device__ __forceinline__ T fsign(T a, T b) { return copysign(fabs(a), b); }

// ---------------------------------------------------------------------------
// horizontal_flux
// One thread per cell, kFluxLevels levels one after the other.  A cell's three faces need four
// triangles (AI = TJ(i,j-1) + TI(i,j), AIJ = TI(i,j) + TJ(i,j), AJ = TJ(i,j) + TI(i-1,j)), formed once
// each from the fields of the six cells they touch, each field loaded once; the cell's weights,
// normals, arc midpoints and areas stay in registers from level to level.  Forming the triangles
// face by face took 72 field loads and 1000 instructions a cell and level; these are 570, and what
// bounds the kernel is the latency of a level's loads at 4 blocks per SM, so each thread asks for its
// own cell's fields of the next level one level ahead (its neighbours' are other threads' own).
// glevel 7, rlevel 1, kall 61 (1.6 GB, 248 us at the copy rate): 642 -> 344 us, 359 of it
// before the outputs took the streaming hint; then 433 without the prefetch, 371 at 3 blocks, 452 with 4
// levels a thread; with the geometry in shared memory 470 and more.
constexpr int kFluxThreads = 128, kFluxLevels = 8;

template <typename T>
struct Vec4 {  // rho, rhovx, rhovy, rhovz of a cell or triangle
  T v[4];
};

// triangle value f0 w1 + f1 w2 + f2 w3 (:146-183); TI(ij) takes (ij, ip1j, ip1jp1), TJ(ij) takes
// (ij, ip1jp1, ijp1)
template <typename T>
__device__ __forceinline__ Vec4<T> tri(const Vec4<T> &f0, const Vec4<T> &f1, const Vec4<T> &f2, const T (&w)[3]) {
  Vec4<T> t;
#pragma unroll
  for (int x = 0; x < 4; ++x) t.v[x] = f0.v[x] * w[0] + f1.v[x] * w[1] + f2.v[x] * w[2];
  return t;
}

template <typename T>
__device__ __forceinline__ void pole_flux(const Dims &D, const FluxIn<T> &in, const FluxOut<T> &out, const Geo<T> &g,
                                          T dt, int l, int k);

// blocks: level blocks fastest (a cell block's geometry is read from L2 after the first), then cell
// blocks, then regions; the last blocks take the poles, one thread per (pole, level)
// FIXED: kFluxLevels levels a thread, known to the compiler (396 us against 427 for glevel 7, rlevel 1,
// kall 61); else lpb.
template <typename T, bool FIXED>
__global__ void __launch_bounds__(kFluxThreads, 4) k_horizontal_flux(Dims D, FluxIn<T> in, FluxOut<T> out, Geo<T> g, T dt,
                                                                  int levels, int nlb, int cellblk, int nmain) {
  const int lpb = FIXED ? kFluxLevels : levels;
  if ((int)blockIdx.x >= nmain) {
    const int t = ((int)blockIdx.x - nmain) * kFluxThreads + (int)threadIdx.x;
    if (t < D.kall * kLallPl) pole_flux(D, in, out, g, dt, t / D.kall, t % D.kall);
    return;
  }
  const int lb = (int)blockIdx.x % nlb, l = (int)blockIdx.x / nlb / cellblk;
  const int ci = (int)blockIdx.x / nlb % cellblk * kFluxThreads + (int)threadIdx.x;
  if (ci >= D.gall) return;
  const int G = D.gall_1d, gmin = D.gmin, gmax = D.gmax;
  const int i = ci % G + 1, j = ci / G + 1;
  const unsigned c = ci;
  const size_t fs = (size_t)D.lall * D.kall * D.gall;  // stride of the last dimension
  const size_t gw = (size_t)D.gall * D.lall, lg = (size_t)l * D.gall;
  const bool sgp = D.have_sgp[l] != 0;
  const T EPS = Num<T>::eps();
  const bool inI = (i >= gmin && i <= gmax), inJ = (j >= gmin && j <= gmax);
  const bool ext = (i >= gmin - 1 && i <= gmax && j >= gmin - 1 && j <= gmax);
  const bool face[3] = {ext && inJ, ext, ext && inI};
  // flx_h(:,4:6) elements no face writes: this cell writes them itself
  const bool in1 = i - 1 >= gmin - 1 && i - 1 <= gmax, jn1 = j - 1 >= gmin - 1 && j - 1 <= gmax;
  const bool own[3] = {!(inJ && in1), !(in1 && jn1), !(inI && jn1)};
  // TI(gmin-1,gmin-1) of a singular region is TJ(gmin,gmin-1) (:188-201): read by the AIJ face of
  // (gmin-1,gmin-1) and the AJ face of (gmin,gmin-1), whose flx_h(gmin,gmin,6) is zero (:311-320)
  const bool singI = sgp && i == gmin - 1 && j == gmin - 1, singJ = sgp && i == gmin && j == gmin - 1;
  T wI[3] = {}, wJ[3] = {}, wJm[3] = {}, wIm[3] = {}, wS[3] = {}, hn[3][3] = {}, xr[3][3] = {}, ra[4] = {};
  if (ext) {
    auto weights = [&](int t, unsigned cell, T (&w)[3]) {
#pragma unroll
      for (int n = 0; n < 3; ++n) w[n] = (g.GMTR_t + ((size_t)(W1 - 1 + n) * 2 + (t - 1)) * gw + lg)[cell];
    };
    weights(TI, c, wI), weights(TJ, c, wJ);
    if (inJ) weights(TJ, c - G, wJm);
    if (inI) weights(TI, c - 1, wIm);
    if (singI) weights(TJ, c + 1, wS);
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        hn[a][x] = (g.GMTR_a + ((size_t)x * 3 + a) * gw + lg)[c];
        xr[a][x] = (g.GRD_xr + ((size_t)x * 3 + a) * gw + lg)[c];
      }
    const T *rarea = g.GMTR_p + (size_t)(P_RAREA - 1) * gw + lg;
    ra[0] = rarea[c], ra[1] = rarea[c + 1], ra[2] = rarea[c + G + 1], ra[3] = rarea[c + G];
  }
  const int k1 = min((lb + 1) * lpb, D.kall);
#pragma unroll 1
  for (int k = lb * lpb; k < k1; ++k) {
    const size_t off = ((size_t)l * D.kall + k) * D.gall;
    auto cell = [&](unsigned p) {
      return Vec4<T>{{(in.rho + off)[p], (in.rhovx + off)[p], (in.rhovy + off)[p], (in.rhovz + off)[p]}};
    };
    if (k + 1 < k1) {
      const size_t on = off + D.gall;
      for (const T *q : {in.rho, in.rhovx, in.rhovy, in.rhovz})
        asm volatile("prefetch.global.L1 [%0];" ::"l"(q + on + c));
    }
    Vec4<T> tI{}, tJ{}, tJm{}, tIm{};
    if (ext) {
      const Vec4<T> f00 = cell(c), f10 = cell(c + 1), f11 = cell(c + G + 1), f01 = cell(c + G);
      Vec4<T> f0m{}, fm0{};
      if (inJ) f0m = cell(c - G);
      if (inI) fm0 = cell(c - 1);
      tI = tri(f00, f10, f11, wI), tJ = tri(f00, f11, f01, wJ);
      tJm = tri(f0m, f10, f00, wJm), tIm = tri(fm0, f00, f01, wIm);
      if (singI) tI = tri(f10, cell(c + G + 2), f11, wS);
      if (singJ) tIm = tJ;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      T *flx = out.flx_h + (size_t)a * fs + off, *fln = out.flx_h + (size_t)(a + 3) * fs + off;
      T f = T(0), x[3] = {T(0), T(0), T(0)};
      if (face[a]) {  // :235-309
        const Vec4<T> &p = (a == 0) ? tJm : (a == 1 ? tI : tJ), &q = (a == 0) ? tI : (a == 1 ? tJ : tIm);
        const T rrhoa2 = T(1) / mx(p.v[0] + q.v[0], EPS);
        const T v[3] = {p.v[1] + q.v[1], p.v[2] + q.v[2], p.v[3] + q.v[3]};
        const T flux = T(0.5) * (v[0] * hn[a][0] + v[1] * hn[a][1] + v[2] * hn[a][2]);
        f = flux * ra[0] * dt;
        const unsigned nb = c + (a == 0 ? 1 : (a == 1 ? G + 1 : G));
        __stcs(fln + nb, (a == 2 && singJ) ? T(0) : -flux * ra[a + 1] * dt);
#pragma unroll
        for (int d = 0; d < 3; ++d) x[d] = xr[a][d] - v[d] * rrhoa2 * dt * T(0.5);
      }
      __stcs(flx + c, f);
#pragma unroll
      for (int d = 0; d < 3; ++d) __stcs(out.GRD_xc + ((size_t)d * 3 + a) * fs + off + c, x[d]);
      if (own[a]) fln[c] = T(0);
    }
  }
}

// one level of a pole (:326-374)
template <typename T>
__device__ __forceinline__ void pole_flux(const Dims &D, const FluxIn<T> &in, const FluxOut<T> &out, const Geo<T> &g,
                                          T dt, int l, int k) {
  const T EPS = Num<T>::eps();
  const size_t off = ((size_t)l * D.kall + k) * kGallPl;
  const size_t fsp = (size_t)kLallPl * D.kall * kGallPl;
  auto GT = [&](int v, int w) { return g.GMTR_t_pl[((size_t)(w - 1) * kLallPl + l) * kGallPl + (v - 1)]; };
  auto GA = [&](int v, int h) { return g.GMTR_a_pl[((size_t)(h - 1) * kLallPl + l) * kGallPl + (v - 1)]; };
  const T rarea = g.GMTR_p_pl[((size_t)(P_RAREA - 1) * kLallPl + l) * kGallPl + 0];
  T rt[7], xt[7], yt[7], zt[7];
  for (int v = 2; v <= 6; ++v) {
    const int vp = (v + 1 == 7) ? 2 : v + 1;
    rt[v] = in.rho_pl[off + 0] * GT(v, W1) + in.rho_pl[off + v - 1] * GT(v, W2) + in.rho_pl[off + vp - 1] * GT(v, W3);
    xt[v] = in.rhovx_pl[off + 0] * GT(v, W1) + in.rhovx_pl[off + v - 1] * GT(v, W2) + in.rhovx_pl[off + vp - 1] * GT(v, W3);
    yt[v] = in.rhovy_pl[off + 0] * GT(v, W1) + in.rhovy_pl[off + v - 1] * GT(v, W2) + in.rhovy_pl[off + vp - 1] * GT(v, W3);
    zt[v] = in.rhovz_pl[off + 0] * GT(v, W1) + in.rhovz_pl[off + v - 1] * GT(v, W2) + in.rhovz_pl[off + vp - 1] * GT(v, W3);
  }
  for (int v = 2; v <= 6; ++v) {
    const int vm = (v - 1 == 1) ? 6 : v - 1;
    const T rr = T(1) / mx(rt[vm] + rt[v], EPS);
    const T vx = xt[vm] + xt[v], vy = yt[vm] + yt[v], vz = zt[vm] + zt[v];
    const T flux = T(0.5) * (vx * GA(v, HNX) + vy * GA(v, HNY) + vz * GA(v, HNZ));
    out.flx_h_pl[off + v - 1] = flux * rarea * dt;
    auto XR = [&](int x) { return g.GRD_xr_pl[((size_t)(x - 1) * kLallPl + l) * kGallPl + (v - 1)]; };
    out.GRD_xc_pl[0 * fsp + off + v - 1] = XR(1) - vx * rr * dt * T(0.5);
    out.GRD_xc_pl[1 * fsp + off + v - 1] = XR(2) - vy * rr * dt * T(0.5);
    out.GRD_xc_pl[2 * fsp + off + v - 1] = XR(3) - vz * rr * dt * T(0.5);
  }
}

// ---------------------------------------------------------------------------
// horizontal_limiter_thuburn

// Qout as the halo fill would leave it, read from where it would copy it: src maps every point
// (regions, then the 12 pole slots) to its source, or to itself; null: Qout is filled already.
template <typename T>
struct HaloSource {
  const int *src;
  const T *Qout;
  __device__ __forceinline__ void load(const Dims &D, const T *Q, const T *Q_pl, int p, int k, T &lo, T &hi) const {
    const int npt = D.lall * D.gall;
    const T *a = p < npt ? Q + ((size_t)(p / D.gall) * D.kall + k) * D.gall + p % D.gall
                         : Q_pl + ((size_t)((p - npt) / kGallPl) * D.kall + k) * kGallPl + (p - npt) % kGallPl;
    lo = a[0];
    hi = a[p < npt ? (size_t)npt * D.kall : (size_t)kLallPl * kGallPl * D.kall];
  }
};

// One thread per (cell, level) in both kernels, the poles in the last blocks of the same launches;
// addresses are a slab base that is the same for the block and a 32-bit offset in the slab.  Bound by
// memory: glevel 7, kall 96 takes 368 us for Qout (104 bytes a cell, 260 us at the copy rate) and 375
// for the apply (120 bytes, 300 us); 486 + 383 us before, and 125 us more for the copy of Qout and
// its halo fill, which the apply now does without.

template <typename T> __device__ __forceinline__ T mn4(T a, T b, T c, T d) { return mn(mn(mn(a, b), c), d); }
template <typename T> __device__ __forceinline__ T mx4(T a, T b, T c, T d) { return mx(mx(mx(a, b), c), d); }

template <typename T>
__device__ __forceinline__ void pole_qout(const Dims &D, const LimIn<T> &in, T *Qout_pl, T *Qin_pl, int l, int k);
template <typename T>
__device__ __forceinline__ void pole_apply(const Dims &D, const LimIn<T> &in, T *q_a_pl, const T *Qout_pl,
                                           const T *Qin_pl, const HaloSource<T> &H, int v, int l, int k);

constexpr int kLimThreads = 128;

// Qout of a cell from the 4-point bounds of its six faces (:152-282).  Faces 4-6 are faces 1-3 of the
// cells (i-1,j), (i-1,j-1), (i,j-1); an interior cell's stencil needs none of the index clamps of
// :152-153.
template <typename T>
__global__ void __launch_bounds__(kLimThreads, 7) k_hlim_qout(Dims D, LimIn<T> in, T *Qout, T *Qout_pl, T *Qin_pl,
                                                           int cellblk, int nmain) {
  if ((int)blockIdx.x >= nmain) {
    const int t = ((int)blockIdx.x - nmain) * kLimThreads + (int)threadIdx.x;
    if (t < D.kall * kLallPl) pole_qout(D, in, Qout_pl, Qin_pl, t / D.kall, t % D.kall);
    return;
  }
  const int ci = (int)blockIdx.x % cellblk * kLimThreads + (int)threadIdx.x, kl = (int)blockIdx.x / cellblk;
  if (ci >= D.gall) return;
  const int l = kl / D.kall, G = D.gall_1d;
  const int i = ci % G + 1, j = ci / G + 1;
  const unsigned c = ci;
  const size_t off = (size_t)kl * D.gall;
  const size_t fs = (size_t)D.lall * D.kall * D.gall;
  const T *q = in.q + off;
  const T q0 = q[c];
  T *Qmin = Qout + off, *Qmax = Qout + fs + off;
  if (i < D.gmin || i > D.gmax || j < D.gmin || j > D.gmax) {  // halo: Qout = q   (:288-301)
    Qmin[c] = q0;
    Qmax[c] = q0;
    return;
  }
  const T *cm1 = in.cmask + off, *cm2 = in.cmask + fs + off, *cm3 = in.cmask + 2 * fs + off;
  const T cc[7] = {T(0), cm1[c], cm2[c], cm3[c], cm1[c - 1], cm2[c - G - 1], cm3[c - G]};
  T ch[7];
#pragma unroll
  for (int f = 1; f <= 6; ++f) ch[f] = (in.ch + (size_t)(f - 1) * fs + off)[c];
  const T dv = (in.d + off)[c];
  const T n1 = q[c + 1], n2 = q[c + G + 1], n3 = q[c + G], n4 = q[c - 1], n5 = q[c - G - 1], n6 = q[c - G];
  const T BIG = Num<T>::big(), EPS = Num<T>::eps();
  const bool sing = i == D.gmin && j == D.gmin && D.have_sgp[l] != 0;  // the AIJ stencil of :192-214
  const T b5 = sing ? q0 : n6, c5 = sing ? n1 : q0;
  const T lo[7] = {T(0), mn4(q0, n6, n1, n2), mn4(q0, n1, n2, n3), mn4(q0, n2, n3, n4),
                   mn4(n4, n5, q0, n3),       mn4(n5, b5, c5, n4), mn4(n6, n1, q0, n5)};
  const T hi[7] = {T(0), mx4(q0, n6, n1, n2), mx4(q0, n1, n2, n3), mx4(q0, n2, n3, n4),
                   mx4(n4, n5, q0, n3),       mx4(n5, b5, c5, n4), mx4(n6, n1, q0, n5)};
  // cmask is 0 or 1 where it comes from a Courant number: an inflow face's bound enters as it is, and an
  // outflow face's, +-BIG, binds nothing and has no part in CQ unless its Courant number says inflow
  bool simple = true, inflow[7];
  T chm[7];
#pragma unroll
  for (int f = 1; f <= 6; ++f) {
    inflow[f] = cc[f] == (f <= 3 ? T(1) : T(0));
    chm[f] = mn(ch[f], T(0));
    simple = simple && (inflow[f] || (cc[f] == (f <= 3 ? T(0) : T(1)) && chm[f] == T(0)));
  }
  T qnext_min = q0, qnext_max = q0, Cin = chm[1], Cout = ch[1] - chm[1], CQmin, CQmax;
#pragma unroll
  for (int f = 2; f <= 6; ++f) Cin = Cin + chm[f], Cout = Cout + ch[f] - chm[f];
  if (simple) {
    CQmin = chm[1] * lo[1], CQmax = chm[1] * hi[1];
#pragma unroll
    for (int f = 1; f <= 6; ++f) {
      qnext_min = (inflow[f] && lo[f] < qnext_min) ? lo[f] : qnext_min;
      qnext_max = (inflow[f] && hi[f] > qnext_max) ? hi[f] : qnext_max;
      if (f > 1) CQmin = CQmin + chm[f] * lo[f], CQmax = CQmax + chm[f] * hi[f];
    }
  } else {
    CQmin = CQmax = T(0);
#pragma unroll
    for (int f = 1; f <= 6; ++f) {
      T qmin, qmax;
      if (f <= 3) {
        qmin = cc[f] * lo[f] + (T(1) - cc[f]) * BIG, qmax = cc[f] * hi[f] + (T(1) - cc[f]) * (-BIG);
      } else {
        qmin = cc[f] * BIG + (T(1) - cc[f]) * lo[f], qmax = cc[f] * (-BIG) + (T(1) - cc[f]) * hi[f];
      }
      qnext_min = mn(qnext_min, qmin), qnext_max = mx(qnext_max, qmax);
      CQmin = (f == 1) ? chm[f] * qmin : CQmin + chm[f] * qmin;
      CQmax = (f == 1) ? chm[f] * qmax : CQmax + chm[f] * qmax;
    }
  }
  const T zerosw = T(0.5) - fsign(T(0.5), fabs(Cout) - EPS), omc = T(1) - Cin - Cout + dv;
  T o[2] = {q0 - CQmax - qnext_max * omc, q0 - CQmin - qnext_min * omc};
  if constexpr (sizeof(T) == 8) quotients(o, recip(Cout + zerosw));
  else o[0] = o[0] / (Cout + zerosw), o[1] = o[1] / (Cout + zerosw);
  Qmin[c] = o[0] * (T(1) - zerosw) + q0 * zerosw;
  Qmax[c] = o[1] * (T(1) - zerosw) + q0 * zerosw;
}

// (:307-367): Qout_pl(n) from the 5 ring faces; Qout_pl(2:6) = 0; keep Qin_pl for the apply
template <typename T>
__device__ __forceinline__ void pole_qout(const Dims &D, const LimIn<T> &in, T *Qout_pl, T *Qin_pl, int l, int k) {
  const T BIG = Num<T>::big(), EPS = Num<T>::eps();
  const size_t off = ((size_t)l * D.kall + k) * kGallPl;
  const size_t fsp = (size_t)kLallPl * D.kall * kGallPl;
  const T *q = in.q_pl + off;
  T qmin1[7], qmax1[7];
  for (int v = 2; v <= 6; ++v) {
    const int vp = (v + 1 == 7) ? 2 : v + 1, vm = (v - 1 == 1) ? 6 : v - 1;
    const T lo = mn(mn(mn(q[0], q[v - 1]), q[vm - 1]), q[vp - 1]);
    const T hi = mx(mx(mx(q[0], q[v - 1]), q[vm - 1]), q[vp - 1]);
    const T c = in.cmask_pl[off + v - 1];
    qmin1[v] = c * lo + (T(1) - c) * BIG;
    qmax1[v] = c * hi + (T(1) - c) * (-BIG);
    // Qin_pl(v,k,l,min/max,1/2)
    Qin_pl[((size_t)0 * 2 + 0) * fsp + off + v - 1] = qmin1[v];
    Qin_pl[((size_t)0 * 2 + 1) * fsp + off + v - 1] = c * BIG + (T(1) - c) * lo;
    Qin_pl[((size_t)1 * 2 + 0) * fsp + off + v - 1] = qmax1[v];
    Qin_pl[((size_t)1 * 2 + 1) * fsp + off + v - 1] = c * (-BIG) + (T(1) - c) * hi;
  }
  T qnmin = q[0], qnmax = q[0];
  for (int v = 2; v <= 6; ++v) {
    qnmin = mn(qnmin, qmin1[v]);
    qnmax = mx(qnmax, qmax1[v]);
  }
  T Cin = 0, Cout = 0, CQmax = 0, CQmin = 0;
  for (int v = 2; v <= 6; ++v) {
    const T chm = in.cmask_pl[off + v - 1] * in.ch_pl[off + v - 1];
    Cin = Cin + chm;
    Cout = Cout - chm + in.ch_pl[off + v - 1];
    CQmin = CQmin + chm * qmin1[v];
    CQmax = CQmax + chm * qmax1[v];
  }
  const T zerosw = T(0.5) - fsign(T(0.5), fabs(Cout) - EPS);
  const T qn = q[0], dn = in.d_pl[off];
  Qout_pl[0 * fsp + off] = (qn - CQmax - qnmax * (T(1) - Cin - Cout + dn)) / (Cout + zerosw) * (T(1) - zerosw) + qn * zerosw;
  Qout_pl[1 * fsp + off] = (qn - CQmin - qnmin * (T(1) - Cin - Cout + dn)) / (Cout + zerosw) * (T(1) - zerosw) + qn * zerosw;
  for (int v = 2; v <= 6; ++v) {
    Qout_pl[0 * fsp + off + v - 1] = T(0);
    Qout_pl[1 * fsp + off + v - 1] = T(0);
  }
}

// (:378-410): cells (i,j) in [gmin-1,gmax]^2, faces 1..3, mirrored to 4..6.  With H.src the halo
// cells' Qout is read from the cells the fill would copy it from, which saves the copy of Qout and
// the fill (a pass over 4 of the kernel's 15 values, and a launch).
template <typename T>
__global__ void __launch_bounds__(kLimThreads) k_hlim_apply(Dims D, LimIn<T> in, T *q_a, T *q_a_pl, const T *Qout,
                                                            const T *Qout_pl, const T *Qin_pl, HaloSource<T> H,
                                                            int cellblk, int nmain) {
  if ((int)blockIdx.x >= nmain) {
    const int t = ((int)blockIdx.x - nmain) * kLimThreads + (int)threadIdx.x, kl = t / 5;
    if (kl < D.kall * kLallPl) pole_apply(D, in, q_a_pl, Qout_pl, Qin_pl, H, t % 5 + 2, kl / D.kall, kl % D.kall);
    return;
  }
  const int ci = (int)blockIdx.x % cellblk * kLimThreads + (int)threadIdx.x, kl = (int)blockIdx.x / cellblk;
  if (ci >= D.gall) return;
  const int l = kl / D.kall, G = D.gall_1d;
  const int i = ci % G + 1, j = ci / G + 1;
  if (i < D.gmin - 1 || i > D.gmax || j < D.gmin - 1 || j > D.gmax) return;
  const unsigned c = ci, nb[3] = {c + 1, c + G + 1, c + G};
  const size_t off = (size_t)kl * D.gall;
  const size_t fs = (size_t)D.lall * D.kall * D.gall;
  const T BIG = Num<T>::big();
  const T *q = in.q + off;
  T cc[3], v[3], os_min, os_max, on_min[3], on_max[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) cc[m] = (in.cmask + m * fs + off)[c], v[m] = (q_a + m * fs + off)[c];
  const T q0 = q[c], n1 = q[nb[0]], n2 = q[nb[1]], n3 = q[nb[2]];
  const T n4 = q[ci > 0 ? c - 1 : 0], n6 = q[ci >= G ? c - G : 0];  // the index clamps of :152-153
  const T *Qmin = Qout + off, *Qmax = Qout + fs + off;
  if (H.src && (i < D.gmin || i == D.gmax || j < D.gmin || j == D.gmax)) {
    const int k = kl % D.kall, *src = H.src + (size_t)l * D.gall;
    H.load(D, Qout, Qout_pl, src[c], k, os_min, os_max);
#pragma unroll
    for (int m = 0; m < 3; ++m) H.load(D, Qout, Qout_pl, src[nb[m]], k, on_min[m], on_max[m]);
  } else {
    os_min = Qmin[c], os_max = Qmax[c];
#pragma unroll
    for (int m = 0; m < 3; ++m) on_min[m] = Qmin[nb[m]], on_max[m] = Qmax[nb[m]];
  }
  T lo[3] = {mn4(q0, n6, n1, n2), mn4(q0, n1, n2, n3), mn4(q0, n2, n3, n4)};
  T hi[3] = {mx4(q0, n6, n1, n2), mx4(q0, n1, n2, n3), mx4(q0, n2, n3, n4)};
  if (i == D.gmin - 1 && j == D.gmin - 1 && D.have_sgp[l] != 0) {  // the singular AIJ stencil of :192-214
    const T ns = q[c + G + 2];
    lo[1] = mn4(q0, n2, ns, n3), hi[1] = mx4(q0, n2, ns, n3);
  }
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const T own_min = cc[m] * lo[m] + (T(1) - cc[m]) * BIG, own_max = cc[m] * hi[m] + (T(1) - cc[m]) * (-BIG);
    const T nb_min = cc[m] * BIG + (T(1) - cc[m]) * lo[m], nb_max = cc[m] * (-BIG) + (T(1) - cc[m]) * hi[m];
    T x = cc[m] * mn(mx(v[m], own_min), own_max) + (T(1) - cc[m]) * mn(mx(v[m], nb_min), nb_max);
    x = cc[m] * mx(mn(x, on_max[m]), on_min[m]) + (T(1) - cc[m]) * mx(mn(x, os_max), os_min);
    (q_a + m * fs + off)[c] = x;
    (q_a + (m + 3) * fs + off)[nb[m]] = x;
  }
}

// (:412-425)
template <typename T>
__device__ __forceinline__ void pole_apply(const Dims &D, const LimIn<T> &in, T *q_a_pl, const T *Qout_pl,
                                           const T *Qin_pl, const HaloSource<T> &H, int v, int l, int k) {
  const size_t off = ((size_t)l * D.kall + k) * kGallPl;
  const size_t fsp = (size_t)kLallPl * D.kall * kGallPl;
  const T c = in.cmask_pl[off + v - 1];
  T x = q_a_pl[off + v - 1], ring_min, ring_max, mid_min, mid_max;
  if (H.src) {
    const int *src = H.src + D.lall * D.gall + l * kGallPl;
    H.load(D, H.Qout, Qout_pl, src[v - 1], k, ring_min, ring_max);
    H.load(D, H.Qout, Qout_pl, src[0], k, mid_min, mid_max);
  } else {
    ring_min = Qout_pl[off + v - 1], ring_max = Qout_pl[fsp + off + v - 1];
    mid_min = Qout_pl[off], mid_max = Qout_pl[fsp + off];
  }
  const T i1min = Qin_pl[((size_t)0 * 2 + 0) * fsp + off + v - 1], i2min = Qin_pl[((size_t)0 * 2 + 1) * fsp + off + v - 1];
  const T i1max = Qin_pl[((size_t)1 * 2 + 0) * fsp + off + v - 1], i2max = Qin_pl[((size_t)1 * 2 + 1) * fsp + off + v - 1];
  x = c * mn(mx(x, i1min), i1max) + (T(1) - c) * mn(mx(x, i2min), i2max);
  x = c * mx(mn(x, ring_max), ring_min) + (T(1) - c) * mx(mn(x, mid_max), mid_min);
  q_a_pl[off + v - 1] = x;
}

// ---------------------------------------------------------------------------
// vertical_limiter_thuburn: one thread per column and kVlimLevels consecutive half levels.  A half
// level needs the Qout of the levels on both sides and nothing else of the column, so the columns
// are cut into chunks that share one Qout at each cut (one in kVlimLevels is formed twice).  With a
// column per thread a glevel-6 grid gave the card 341 blocks and a chain of 40 dependent levels
// (69 us, and 56 us more for the 12 pole columns in a launch behind it).  Now 23 us there, of the 13.5
// its 88 MB need (4 levels a thread 25, 13 levels 28), and 170 us for glevel 7, kall 96 (0.78 GB, 120 us).
constexpr int kVlimLevels = 8, kVlimThreads = 128;

template <typename T>
struct VlimLevel {  // what Qout of a level reads: its own values and q and ck1 around it
  T q, d, c1, c2;
};
template <typename T, bool POLE>
__device__ __forceinline__ void vlim_qout(T qm, const VlimLevel<T> &v, T qp, T c1p, T &inflagL, T &Qmin, T &Qmax) {
  const T BIG = Num<T>::big(), EPS = Num<T>::eps();
  inflagL = T(0.5) - fsign(T(0.5), v.c1);
  const T inflagU = T(0.5) + fsign(T(0.5), c1p);
  const T qk = v.q, c1 = v.c1, c2 = v.c2;
  const T minL = mn(qk, qm) + (T(1) - inflagL) * BIG;
  const T minU = mn(qk, qp) + (T(1) - inflagU) * BIG;
  const T maxL = mx(qk, qm) - (T(1) - inflagL) * BIG;
  const T maxU = mx(qk, qp) - (T(1) - inflagU) * BIG;
  const T qnmin = mn(mn(minL, minU), qk);
  const T qnmax = mx(mx(maxL, maxU), qk);
  const T Cin = inflagL * c1 + inflagU * c2;
  const T Cout = (T(1) - inflagL) * c1 + (T(1) - inflagU) * c2;
  T CQmin, CQmax;
  if (POLE) {  // the pole loop groups ck*Qin first (:212-215)
    CQmax = inflagL * (c1 * maxL) + inflagU * (c2 * maxU);
    CQmin = inflagL * (c1 * minL) + inflagU * (c2 * minU);
  } else {
    CQmin = inflagL * c1 * minL + inflagU * c2 * minU;
    CQmax = inflagL * c1 * maxL + inflagU * c2 * maxU;
  }
  const T zerosw = T(0.5) - fsign(T(0.5), fabs(Cout) - EPS);
  T o[2] = {(qk - qnmax) + qnmax * (Cin + Cout - v.d) - CQmax, (qk - qnmin) + qnmin * (Cin + Cout - v.d) - CQmin};
  if constexpr (sizeof(T) == 8) quotients(o, recip(Cout + zerosw));
  else o[0] = o[0] / (Cout + zerosw), o[1] = o[1] / (Cout + zerosw);
  Qmin = o[0] * (T(1) - zerosw) + qk * zerosw;
  Qmax = o[1] * (T(1) - zerosw) + qk * zerosw;
}

// half levels [k0, k0 + kVlimLevels) (0-based, below kmax) of one column; arrays at the column's
// first level, g elements from level to level, ck2 at ck + ck2off.  Levels kmin - 1 and kmax + 1
// lie inside the arrays of a grid with ghost levels; without them the nearest level is read.
template <typename T, bool POLE>
__device__ __forceinline__ void vlim_chunk(unsigned g, int k0, int kmax, int kall, T *qh, const T *q, const T *d,
                                           const T *ck, size_t ck2off) {
  const T *ck2 = ck + ck2off;
  const int k1 = min(k0 + kVlimLevels, kmax);
  auto at = [&](int k) { return (unsigned)min(max(k, 0), kall - 1) * g; };
  auto level = [&](int k) { return VlimLevel<T>{q[at(k)], d[at(k)], ck[at(k)], ck2[at(k)]}; };
  VlimLevel<T> m = level(k0 - 1), v = level(k0);
  T qp = q[at(k0 + 1)], c1p = ck[at(k0 + 1)], qm = q[at(k0 - 2)], fl, Qmin_m, Qmax_m;
  vlim_qout<T, POLE>(qm, m, v.q, v.c1, fl, Qmin_m, Qmax_m);
  qm = m.q;
#pragma unroll 4
  for (int k = k0; k < k1; ++k) {
    VlimLevel<T> n{qp, T(0), c1p, T(0)};
    T qn = T(0), c1n = T(0);
    if (k + 1 < k1) {  // the next level's inputs
      n.d = d[at(k + 1)], n.c2 = ck2[at(k + 1)];
      qn = q[at(k + 2)], c1n = ck[at(k + 2)];
    }
    T &o = qh[at(k)];
    const T h = o;
    T inflagL, Qmin, Qmax;
    vlim_qout<T, POLE>(qm, v, qp, c1p, inflagL, Qmin, Qmax);
    o = inflagL * mx(mn(h, Qmax_m), Qmin_m) + (T(1) - inflagL) * mx(mn(h, Qmax), Qmin);
    Qmin_m = Qmin, Qmax_m = Qmax;
    qm = v.q, v = n, qp = qn, c1p = c1n;
  }
}

// blocks: column blocks of a region fastest, then its chunks, then the regions; the last blocks take
// the pole columns
template <typename T>
__global__ void __launch_bounds__(kVlimThreads) k_vlim(Dims D, int nchunk, int colblk, int nmain, T *q_h, const T *q,
                                                       const T *d, const T *ck, T *q_h_pl, const T *q_pl,
                                                       const T *d_pl, const T *ck_pl) {
  const int b = blockIdx.x;
  if (b < nmain) {
    const int u = b % colblk * kVlimThreads + (int)threadIdx.x;
    if (u >= D.gall) return;
    const int l = b / colblk / nchunk, k0 = D.kmin + b / colblk % nchunk * kVlimLevels;  // 0-based kmin+1 ..
    const size_t base = (size_t)l * D.kall * D.gall + u;
    vlim_chunk<T, false>(D.gall, k0, D.kmax, D.kall, q_h + base, q + base, d + base, ck + base,
                         (size_t)D.lall * D.kall * D.gall);
    return;
  }
  const int t = (b - nmain) * kVlimThreads + (int)threadIdx.x;
  if (t >= kLallPl * kGallPl * nchunk) return;
  const int col = t % (kLallPl * kGallPl), k0 = D.kmin + t / (kLallPl * kGallPl) * kVlimLevels;
  const size_t base = (size_t)(col / kGallPl) * D.kall * kGallPl + col % kGallPl;
  vlim_chunk<T, true>(kGallPl, k0, D.kmax, D.kall, q_h_pl + base, q_pl + base, d_pl + base, ck_pl + base,
                      (size_t)kLallPl * D.kall * kGallPl);
}

// ---------------------------------------------------------------------------
// halo/pole fill as one gather: var(dst) = var(src) for every (entry, k, v), of one array or of two
// (a step's rhogq and rhog).  A thread takes one entry through kGatherPlanes (k, v) planes: the
// points' addresses are worked out once and that many loads are in flight.  Bound by DRAM
// sectors: a point of a region's i-edge column costs 64 bytes read and 64 written for its 16.  One element
// a thread -> 4 planes: 143 -> 122 us (glevel 7, kall 96, 16 arrays), 298 -> 255 (glevel 8), 13.6 -> 11.6
// (glevel 6, kall 42, 8 arrays); 8 and 16 planes were slower.
constexpr int kGatherThreads = 128, kGatherPlanes = 4;

template <typename T>
__global__ void __launch_bounds__(kGatherThreads) k_gather(int nent, const int *__restrict__ dst,
                                                           const int *__restrict__ src, int entblk, int gall, int lall,
                                                           int kmax, int vmax, int planes, T *var, T *var_pl, T *var2,
                                                           T *var2_pl) {
  const int e = (int)blockIdx.x % entblk * kGatherThreads + (int)threadIdx.x;
  const int p0 = (int)blockIdx.x / entblk * kGatherPlanes, n = min(kGatherPlanes, planes - p0);
  if (e >= nent) return;
  const int npt = lall * gall, pd = dst[e], ps = src[e];
  const bool dpl = pd >= npt, spl = ps >= npt;
  // the points' offsets at level 0 of a variable, and their steps from level to level
  auto offset = [&](int p) {
    return p < npt ? (size_t)(p / gall) * kmax * gall + p % gall
                   : (size_t)((p - npt) / kGallPl) * kmax * kGallPl + (p - npt) % kGallPl;
  };
  const size_t od = offset(pd), os = offset(ps), kd = dpl ? kGallPl : gall, ks = spl ? kGallPl : gall;
  const size_t vr = (size_t)npt * kmax, vp = (size_t)kLallPl * kGallPl * kmax;  // a variable of var and of var_pl
  int k = p0 % kmax, v = p0 / kmax;  // variable vmax is var2
  T x[kGatherPlanes], *to[kGatherPlanes];
#pragma unroll
  for (int u = 0; u < kGatherPlanes; ++u)
    if (u < n) {
      T *r = v < vmax ? var + v * vr : var2, *p = v < vmax ? var_pl + v * vp : var2_pl;
      to[u] = (dpl ? p : r) + od + k * kd;
      x[u] = ((spl ? p : r) + os)[k * ks];
      if (++k == kmax) k = 0, ++v;
    }
#pragma unroll
  for (int u = 0; u < kGatherPlanes; ++u)
    if (u < n) *to[u] = x[u];
}

// ---------------------------------------------------------------------------
// launchers
template <typename T>
void launch_horizontal_flux(const Dims &D, const FluxIn<T> &in, const FluxOut<T> &out, const Geo<T> &g, T dt,
                            cudaStream_t s) {
  const int cellblk = (D.gall + kFluxThreads - 1) / kFluxThreads;
  // a grid whose levels fit one wave (4 blocks on each of 148 SMs) in runs of at most 12 takes that
  // split: 130 x 130 x 42 in one region, 38.4 us a call at 11 levels against 40.2 at 8 (1.35 waves).
  // Where not one level fits (fit = 0) there is no such split, and runs of 8 in the fixed form are the
  // faster ones: glevel 7, kall 7, 9 and 12 take 54, 68 and 81 us, in one run of all levels 59, 72
  // and 92; glevel 8, kall 6 and 12 150 and 287 against 160 and 296, kall 9 (runs of 8 and 1) 231 against 226
  const int fit = 4 * 148 / (cellblk * D.lall), one = fit > 0 ? (D.kall + fit - 1) / fit : 0;
  const int lpb = fit > 0 && one <= 12 ? one : kFluxLevels;
  const int nlb = (D.kall + lpb - 1) / lpb;
  const int nmain = nlb * cellblk * D.lall;
  const int npole = D.have_pl ? (D.kall * kLallPl + kFluxThreads - 1) / kFluxThreads : 0;
  auto kernel = lpb == kFluxLevels ? k_horizontal_flux<T, true> : k_horizontal_flux<T, false>;
  kernel<<<(unsigned)(nmain + npole), kFluxThreads, 0, s>>>(D, in, out, g, dt, lpb, nlb, cellblk, nmain);
}

template <typename T>
void launch_hlim_qout(const Dims &D, const LimIn<T> &in, T *Qout, T *Qout_pl, T *Qin_pl, cudaStream_t s) {
  const int cellblk = (D.gall + kLimThreads - 1) / kLimThreads, nmain = cellblk * D.kall * D.lall;
  const int npole = D.have_pl ? (D.kall * kLallPl + kLimThreads - 1) / kLimThreads : 0;
  k_hlim_qout<T><<<(unsigned)(nmain + npole), kLimThreads, 0, s>>>(D, in, Qout, Qout_pl, Qin_pl, cellblk, nmain);
}

template <typename T>
void launch_hlim_apply(const Dims &D, const LimIn<T> &in, T *q_a, T *q_a_pl, const T *Qout, const T *Qout_pl,
                       const T *Qin_pl, const int *halo_src, cudaStream_t s) {
  const int cellblk = (D.gall + kLimThreads - 1) / kLimThreads, nmain = cellblk * D.kall * D.lall;
  const int npole = D.have_pl ? (D.kall * kLallPl * 5 + kLimThreads - 1) / kLimThreads : 0;
  k_hlim_apply<T><<<(unsigned)(nmain + npole), kLimThreads, 0, s>>>(D, in, q_a, q_a_pl, Qout, Qout_pl, Qin_pl,
                                                                    HaloSource<T>{halo_src, Qout}, cellblk, nmain);
}

template <typename T>
void launch_vlim(const Dims &D, T *q_h, T *q_h_pl, const T *q, const T *q_pl, const T *d, const T *d_pl,
                 const T *ck, const T *ck_pl, cudaStream_t s) {
  if (D.kmax <= D.kmin) return;
  const int nchunk = (D.kmax - D.kmin + kVlimLevels - 1) / kVlimLevels;
  const int colblk = (D.gall + kVlimThreads - 1) / kVlimThreads, nmain = colblk * nchunk * D.lall;
  const int npole = D.have_pl ? (kLallPl * kGallPl * nchunk + kVlimThreads - 1) / kVlimThreads : 0;
  k_vlim<T><<<(unsigned)(nmain + npole), kVlimThreads, 0, s>>>(D, nchunk, colblk, nmain, q_h, q, d, ck, q_h_pl, q_pl,
                                                               d_pl, ck_pl);
}

template <typename T>
void launch_gather(const Dims &D, int nent, const int *dst, const int *src, int kmax, int vmax, T *var, T *var_pl,
                   cudaStream_t s, T *var2, T *var2_pl) {
  const int planes = kmax * (vmax + (var2 ? 1 : 0));
  if (nent == 0 || planes == 0) return;
  const int entblk = (nent + kGatherThreads - 1) / kGatherThreads, chunks = (planes + kGatherPlanes - 1) / kGatherPlanes;
  k_gather<T><<<(unsigned)(entblk * chunks), kGatherThreads, 0, s>>>(nent, dst, src, entblk, D.gall, D.lall, kmax, vmax,
                                                                     planes, var, var_pl, var2, var2_pl);
}

#define INSTANTIATE(T)                                                                                        \
  template void launch_horizontal_flux<T>(const Dims &, const FluxIn<T> &, const FluxOut<T> &, const Geo<T> &, \
                                          T, cudaStream_t);                                                   \
  template void launch_hlim_qout<T>(const Dims &, const LimIn<T> &, T *, T *, T *, cudaStream_t);             \
  template void launch_hlim_apply<T>(const Dims &, const LimIn<T> &, T *, T *, const T *, const T *,          \
                                     const T *, const int *, cudaStream_t);                                                \
  template void launch_vlim<T>(const Dims &, T *, T *, const T *, const T *, const T *, const T *, const T *, \
                               const T *, cudaStream_t);                                                      \
  template void launch_gather<T>(const Dims &, int, const int *, const int *, int, int, T *, T *, cudaStream_t, \
                                 T *, T *);
INSTANTIATE(double)
INSTANTIATE(float)

}  // namespace icoadv
