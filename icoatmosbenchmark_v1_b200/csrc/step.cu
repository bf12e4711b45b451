// The composed tracer step, plain FP64 path: the reference kernels' operations
// with the pieces the reference leaves out (Courant numbers, gradient, remap,
// rhogq update, vertical flux), fused into three launches per group of tracers
// (below).  The FP32 / FP64 batched path is fast_kernels.cu.
//
// The composition (horizontal sub-step, then vertical sub-step, then the halo
// fill of the state) and every formula match the CPU oracle's definition of
// the step; compiled with --fmad=false the FP64 results of a finite state equal
// it bit for bit.
//
//   ch    = flx_h / rhog,  cmask = 0.5 - sign(0.5, ch - EPS)
//   q     = rhogq / rhog
//   grad  = sum_n coef_grad(n) q(nb_n)   (stencil of dyn_metrics/src/mod_oprt.f90:499-734)
//   q_a   = q(up) + grad(up).(GRD_xc - GRD_x(up)), blended by cmask (Miura 2007 remap,
//           docs/NICAM/src/20_intro_nicam.tex:368-429)
//   q_a   = horizontal_limiter_thuburn(q_a, q, 0, ch, cmask) with the Qout halo fill
//   rhogq -= sum_m flx_h(m) q_a(m);  rhog -= sum_m flx_h(m)
//   vertical: ck from rhogw, q_h by linear interpolation, vertical_limiter_thuburn,
//           rhogq -= d/dz(rhogw q_h) dt, rhog -= d/dz(rhogw) dt
#include <cuda_runtime.h>

#include <cfloat>
#include <type_traits>

#include "plain_cells.cuh"

namespace icoadv {

// ---------------------------------------------------------------------------
// The step itself: the tracers go through in groups of up to kPlainGroup, three launches a group.
//
//   k_plain_cells  one thread per interior cell, a tile's levels and tracers streamed through: the
//                  gradient, Qout and the 4-point bounds of the cell's six faces from q in shared
//                  memory, and the limited value of each of its outflow faces (the faces whose
//                  upwind cell it is), which needs nothing but what the thread then holds.  Gradient
//                  and Qout go to memory at region-boundary cells and pole centres only (bb), the
//                  values halo cells stand for.
//   k_plain_seam   the limited value of the faces with a halo cell on one side, per region as the
//                  reference computes them (each side in its own index frame), from bb.
//   k_plain_column rhogq after the horizontal sub-step, formed level by level from the six face
//                  values, and the vertical sub-step of the column as it streams by, in place.
//
// A face value travels once through memory (24 bytes written and read per update); gradient,
// remap value, Courant number, mask and Qout never do.  Against one launch per piece and tracer
// (14 launches a tracer, a column's levels in local memory): 9.90 -> 3.17 ms for glevel 7, kall 61,
// 5 tracers, 1.59 -> 0.30 ms for glevel 5, kall 42, 8 tracers.  Every value is the result of the
// reference's operation sequence; where the reference blends two sides by a mask of 0 or 1
// (c a + (1 - c) b), the chosen side is taken, which is the same number while both are finite.
// A state that holds a NaN or an infinity keeps one there, but its faces' other cells get it only
// where the face's flow or bounds bring it; the blend (0 * NaN) handed it upwind as well.
constexpr int kTileCells = 256;  // threads of k_plain_cells: one per cell of a TX x (256 / TX) tile
constexpr int kCellBlocks = 2;   // its blocks per SM: 128 registers a thread, which hold one tracer's values

// pole centre (p, k) of tracer t: gradient and Qout (mod_src_tracer.f90:307-367) into bb
__device__ __forceinline__ void pole_centre(const PlainArgs &P, int t, int p, int k) {
  const double BIG = DBL_MAX;
  const size_t off = ((size_t)p * P.D.kall + k) * kGallPl;
  double q[kGallPl];
  for (int v = 0; v < kGallPl; ++v) q[v] = P.Qp[t * P.n3p() + off + v] / P.rhop[off + v];
  double *o = P.bval(t, k, P.nb - 2 + p);
  for (int x = 0; x < 3; ++x) {
    const double *cx = P.cgp + ((size_t)p * 3 + x) * 6;
    double s = cx[0] * q[0];
    for (int v = 1; v < 6; ++v) s = s + cx[v] * q[v];
    o[x] = s;
  }
  double qnmin = q[0], qnmax = q[0], Cin = 0, Cout = 0, CQmax = 0, CQmin = 0;
  for (int v = 1; v <= 5; ++v) {
    const int vp = (v == 5) ? 1 : v + 1, vm = (v == 1) ? 5 : v - 1;
    const double ch = P.flxp[off + v] / P.rhop[off];
    const double c = upmask(P.flxp[off + v], P.rhop[off]) ? 1.0 : 0.0;
    const double qmin = c * mn4(q[0], q[v], q[vm], q[vp]) + (1.0 - c) * BIG;
    const double qmax = c * mx4(q[0], q[v], q[vm], q[vp]) + (1.0 - c) * (-BIG);
    qnmin = mn(qnmin, qmin), qnmax = mx(qnmax, qmax);
    const double chm = c * ch;
    Cin = Cin + chm;
    Cout = Cout - chm + ch;
    CQmin = CQmin + chm * qmin;
    CQmax = CQmax + chm * qmax;
  }
  const double zsw = 0.5 - sgn(0.5, fabs(Cout) - DBL_EPSILON), dn = 0.0;
  o[3] = (q[0] - CQmax - qnmax * (1.0 - Cin - Cout + dn)) / (Cout + zsw) * (1.0 - zsw) + q[0] * zsw;
  o[4] = (q[0] - CQmin - qnmin * (1.0 - Cin - Cout + dn)) / (Cout + zsw) * (1.0 - zsw) + q[0] * zsw;
}

// Bound by instruction issue and latency: 1.67 ms of the 3.17, of which the set-up of a level (620
// instructions a cell against 550 per tracer) is a third.  One tracer per pass of the loop and two
// blocks per SM keep every value in registers; two tracers, or three blocks, spill and take 2.5-2.6
// ms.  The next level's set-up inputs are asked for while a level's tracers go through (1.72 without).
// grid: blocks 0 .. ntile*nlb-1 (level block fastest: a tile's gradient coefficients come from L2
// after the first), then the pole centres
template <int TX>
__global__ void __launch_bounds__(kTileCells, kCellBlocks) k_plain_cells(PlainArgs P, int ntx, int nty, int nlb, int lpb) {
  using Tile = CellTile<TX, kTileCells>;
  using S = typename Tile::Smem;
  extern __shared__ __align__(16) unsigned char raw[];
  S &s = *reinterpret_cast<S *>(raw);
  const Dims &D = P.D;
  const int G = D.gall_1d, tid = threadIdx.x;
  const int nmain = ntx * nty * D.lall * nlb;
  if ((int)blockIdx.x >= nmain) {
    const int u = ((int)blockIdx.x - nmain) * kTileCells + tid;
    if (u < P.nt * kLallPl * D.kall) pole_centre(P, u / (kLallPl * D.kall), u / D.kall % kLallPl, u % D.kall);
    return;
  }
  const int lb = (int)blockIdx.x % nlb;
  Tile T;
  T.init(P, s, (int)blockIdx.x / nlb, ntx, nty);
  const int c = T.c;
  const size_t n3 = P.n3();
  const int kfirst = D.kmin - 1, kend = D.kmax;  // physical levels, 0-based
  const int k0 = kfirst + lb * lpb, k1 = min(k0 + lpb, kend);
  for (int k = k0; k < k1; ++k) {
    const size_t off = ((size_t)T.l * D.kall + k) * D.gall;
    double Qw[Tile::NSLOT][1];
    const double *Qs = P.Q + off;
    auto load = [&] {
#pragma unroll
      for (int r = 0; r < Tile::NSLOT; ++r)
        if (T.has(r)) Qw[r][0] = Qs[T.wc[r]];
    };
    load();  // with the level's other global loads, before the first wait
    Recip rw[Tile::NSLOT];
    CellFlow F;
    double flx[6];
    T.level(P, s, off, rw, F, flx);
    if (k + 1 < k1) T.prefetch(P, off + D.gall);
    // ---- the tracers; their q alternates between two buffers
    double *fv = P.fv + off;
    for (int t = 0; t < P.nt; ++t, fv += 3 * n3) {
      const int b = t & 1;
#pragma unroll
      for (int r = 0; r < Tile::NSLOT; ++r)
        if (T.has(r)) {
          quotients(Qw[r], rw[r]);
          s.q[b][tid + r * kTileCells] = Qw[r][0];
        }
      Qs += n3;
      if (t + 1 < P.nt) load();
      __syncthreads();
      double n[7], g[3];
      T.gradient(s, b, n, g);
      CellLimits L;
      cell_limits(n, F, T.sing, L);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const bool f = (F.side >> a) & 1u;
        double v = n[0];
#pragma unroll
        for (int d = 0; d < 3; ++d) v = v + g[d] * s.disp[a * 3 + d][F.sl[a]];
        v = mn(mx(v, f ? L.lo[a + 4] : L.lo[a + 1]), f ? L.hi[a + 4] : L.hi[a + 1]);
        v = mx(mn(v, L.Qmax), L.Qmin);
        store_if(F.st[a] >= 0, fv + a * n3 + F.st[a], v);
      }
      if (F.again) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
          if ((F.again >> a) & 1u) {
            double v = n[0];
#pragma unroll
            for (int d = 0; d < 3; ++d) v = v + g[d] * s.disp[a * 3 + d][T.ow - Tile::slot_back(a)];
            v = mn(mx(v, L.lo[a + 4]), L.hi[a + 4]);
            (fv + a * n3)[c - face_step(a, G)] = mx(mn(v, L.Qmax), L.Qmin);
          }
      }
      if (T.bs >= 0) {
        double *o = P.bval(t, k, T.bs);
        o[0] = g[0], o[1] = g[1], o[2] = g[2], o[3] = L.Qmin, o[4] = L.Qmax;
      }
    }
  }
}

// Faces with a halo cell on one side: one thread per (seam face, level), the tracers one after the other
// with the next one's inputs in flight.  The face's cells, upwind side, displacement and the
// reciprocals of rhog are formed once (a thread per tracer took five divisions each: 143 -> 80 us for
// glevel 7, kall 61, 5 tracers, 30 -> 22 for glevel 5, kall 42, 8).
__global__ void __launch_bounds__(128) k_plain_seam(PlainArgs P) {
  const Dims &D = P.D;
  const long long u = (long long)blockIdx.x * 128 + threadIdx.x;
  if (u >= (long long)P.ns * (D.kmax - D.kmin + 1)) return;
  const int e = (int)(u % P.ns), k = D.kmin - 1 + (int)(u / P.ns);
  const int code = P.seam[e], G = D.gall_1d;
  const int a = code % 3, o = code / 3 % D.gall, l = code / 3 / D.gall;
  const int i = o % G + 1, j = o / G + 1, nb = o + face_step(a, G);
  const bool inO = P.inner(i, j), inN = P.inner(a < 2 ? i + 1 : i, a > 0 ? j + 1 : j);
  if (!inO && !inN) return;  // no interior cell reads it
  const size_t n3 = P.n3(), off = ((size_t)l * D.kall + k) * D.gall, gw = (size_t)D.lall * D.gall;
  const double *rho = P.rho + off;
  // the face's 4 points, owner first (mod_src_tracer.f90:152-214); nb is the third, at the singular
  // point the second
  const bool sing = a == 1 && D.have_sgp[l] != 0 && i == D.gmin - 1 && j == D.gmin - 1;
  int p[4] = {o, o + 1, o + G + 1, o + G};
  if (a == 0) p[1] = max(o - G, 0), p[2] = o + 1, p[3] = o + G + 1;
  else if (a == 2) p[1] = o + G + 1, p[2] = o + G, p[3] = max(o - 1, 0);
  else if (sing) p[1] = o + G + 1, p[2] = o + G + 2, p[3] = o + G;
  Recip r[4];
#pragma unroll
  for (int n = 0; n < 4; ++n) r[n] = recip(rho[p[n]]);
  const bool cm = upmask(P.flx[(size_t)a * n3 + off + o], r[0].b);
  const int up = cm ? nb : o, b = P.bsrc[(size_t)l * D.gall + up];
  double disp[3];
#pragma unroll
  for (int d = 0; d < 3; ++d)
    disp[d] = P.xc[((size_t)d * 3 + a) * n3 + off + o] - P.GRD_x[d * gw + (size_t)l * D.gall + up];
  const double *Q = P.Q + off, *bv = P.bval(0, k, b >= 0 ? b : 0);
  double *fv = P.fv + (size_t)a * n3 + off + o;
  const size_t bs = (size_t)D.kall * P.nb * 5;
  double Qn[4], bn[5];
  auto fetch = [&] {
#pragma unroll
    for (int n = 0; n < 4; ++n) Qn[n] = Q[p[n]];
    if (b >= 0) {
#pragma unroll
      for (int x = 0; x < 5; ++x) bn[x] = bv[x];
    }
    Q += n3, bv += bs;
  };
  fetch();
  for (int t = 0; t < P.nt; ++t, fv += 3 * n3) {
    double q[4][1], g[5];
#pragma unroll
    for (int n = 0; n < 4; ++n) q[n][0] = Qn[n];
#pragma unroll
    for (int x = 0; x < 5; ++x) g[x] = bn[x];
    if (t + 1 < P.nt) fetch();
#pragma unroll
    for (int n = 0; n < 4; ++n) quotients(q[n], r[n]);
    const double qu = !cm ? q[0][0] : (sing ? q[1][0] : q[2][0]);
    if (b < 0) g[0] = g[1] = g[2] = 0.0, g[3] = g[4] = qu;  // a halo point no list fills: no gradient, Qout = q
    double v = qu;
#pragma unroll
    for (int d = 0; d < 3; ++d) v = v + g[d] * disp[d];
    v = mn(mx(v, mn4(q[0][0], q[1][0], q[2][0], q[3][0])), mx4(q[0][0], q[1][0], q[2][0], q[3][0]));
    *fv = mx(mn(v, g[4]), g[3]);
  }
}

// Vertical limiter (dyn_vert_adv_limiter/src/mod_src_tracer.f90:107-186, d = 0): the
// tracer-independent part of a level and one tracer's Qout.
struct VPar {
  double infl, bl, bu, a1, a2, icm, zsw;
  Recip den;
};
__device__ __forceinline__ VPar vpar(double c1, double c2, double c1u) {
  VPar v;
  v.infl = 0.5 - sgn(0.5, c1);
  const double infu = 0.5 + sgn(0.5, c1u), dv = 0.0;
  v.bl = (1.0 - v.infl) * DBL_MAX, v.bu = (1.0 - infu) * DBL_MAX;
  v.a1 = v.infl * c1, v.a2 = infu * c2;
  const double Cin = v.a1 + v.a2, Cout = (1.0 - v.infl) * c1 + (1.0 - infu) * c2;
  v.zsw = 0.5 - sgn(0.5, fabs(Cout) - DBL_EPSILON);
  v.den = recip(Cout + v.zsw);
  v.icm = Cin + Cout - dv;
  return v;
}
__device__ __forceinline__ void vqout(const VPar &v, double qm, double qk, double qp, double &Qmin, double &Qmax) {
  const double minL = mn(qk, qm) + v.bl, minU = mn(qk, qp) + v.bu;
  const double maxL = mx(qk, qm) - v.bl, maxU = mx(qk, qp) - v.bu;
  const double qnmin = mn(mn(minL, minU), qk), qnmax = mx(mx(maxL, maxU), qk);
  const double CQmin = v.a1 * minL + v.a2 * minU, CQmax = v.a1 * maxL + v.a2 * maxU;
  double o[2] = {(qk - qnmax) + qnmax * v.icm - CQmax, (qk - qnmin) + qnmin * v.icm - CQmin};
  quotients(o, v.den);
  Qmin = o[0] * (1.0 - v.zsw) + qk * v.zsw;
  Qmax = o[1] * (1.0 - v.zsw) + qk * v.zsw;
}
__device__ __forceinline__ double vclamp(double infl, double h, double mnL, double mxL, double mnU, double mxU) {
  const double a1 = (h < mxL) ? h : mxL, b1 = (mnL > a1) ? mnL : a1;
  const double a2 = (h < mxU) ? h : mxU, b2 = (mnU > a2) ? mnU : a2;
  return infl * b1 + (1.0 - infl) * b2;
}

constexpr int kColThreads = 128, kColStages = 2, kColBlocks = 3;
constexpr int kColSmem = kColStages * (8 + 7 * 2) * kColThreads * (int)sizeof(double);

__device__ __forceinline__ void copy_async(double *dst, const double *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// the two sub-steps of one pole column (p, tracer t): a thread per level, every stage level-parallel
__device__ __forceinline__ void pole_column(const PlainArgs &P, int p, int t) {
  extern __shared__ __align__(16) double ring[];  // the memory of the other blocks' input stages
  double *sq = ring, *sh = sq + kColThreads, *s1 = sh + kColThreads, *s2 = s1 + kColThreads, *smn = s2 + kColThreads,
         *smx = smn + kColThreads;
  const Dims &D = P.D;
  const int K = D.kall, k = threadIdx.x, kmin = D.kmin - 1, kmax = D.kmax - 1;
  const size_t off = ((size_t)p * K + k) * kGallPl, n3p = P.n3p();
  double *Q = P.Qp + (size_t)t * n3p;
  const bool phys = k >= kmin && k <= kmax;
  double Qh = 0.0, r = 1.0;
  if (k < K) {
    double rs = P.flxp[off + 1];
    for (int v = 2; v <= 5; ++v) rs = rs + P.flxp[off + v];
    r = P.rhop[off] - rs;
  }
  if (phys) {  // rhogq after the horizontal sub-step: the five ring faces
    double q[kGallPl], s = 0.0;
    for (int v = 0; v < kGallPl; ++v) q[v] = Q[off + v] / P.rhop[off + v];
    const double *bc = P.bval(t, k, P.nb - 2 + p);
    for (int v = 1; v <= 5; ++v) {
      const int vp = (v == 5) ? 1 : v + 1, vm = (v == 1) ? 5 : v - 1;
      const bool c = upmask(P.flxp[off + v], P.rhop[off]);
      const int up = c ? v : 0;
      const double *bv = c ? P.bval(t, k, P.ring[p * kVlink + v - 1]) : bc;
      double f = q[up];
      for (int d = 0; d < 3; ++d)
        f = f + bv[d] * (P.xcp[d * n3p + off + v] - P.GRD_xp[((size_t)d * kLallPl + p) * kGallPl + up]);
      f = mn(mx(f, mn4(q[0], q[v], q[vm], q[vp])), mx4(q[0], q[v], q[vm], q[vp]));
      f = mx(mn(f, bv[4]), bv[3]);
      s = (v == 1) ? P.flxp[off + v] * f : s + P.flxp[off + v] * f;
    }
    Qh = Q[off] - s;
  }
  if (K == 1) {
    if (k == 0) Q[off] = Qh;
    return;
  }
  auto W = [&](int kk) { return P.wp[((size_t)p * K + kk) * kGallPl]; };
  double c1 = 0.0, c2 = 0.0;
  if (phys || k == K - 1) c1 = -W(k) * P.dt * P.rdgz[k] / r;
  if (phys) c2 = W(k + 1) * P.dt * P.rdgz[k] / r;
  if (k < K) s1[k] = c1, s2[k] = c2;
  if (phys) {
    const double qk = Qh / r;
    sq[k] = qk;
    if (k == kmin) sq[0] = qk;
    if (k == kmax) sq[K - 1] = qk;
  }
  __syncthreads();
  double h = (k >= kmin && k < K) ? P.afact[k] * sq[k] + P.bfact[k] * sq[k - 1] : 0.0, infl = 0.0;
  if (phys) {
    const VPar v = vpar(s1[k], s2[k], s1[k + 1]);
    infl = v.infl;
    vqout(v, sq[k - 1], sq[k], sq[k + 1], smn[k], smx[k]);
  }
  __syncthreads();
  if (phys && k > kmin) h = vclamp(infl, h, smn[k - 1], smx[k - 1], smn[k], smx[k]);
  if (k < K) sh[k] = h;
  __syncthreads();
  if (phys) {
    const double fu = W(k + 1) * sh[k + 1], fl = W(k) * sh[k];
    const double Qn = Qh - (fu - fl) * P.dt * P.rdgz[k];
    Q[off] = Qn;
    if (k == kmin) Q[(size_t)p * K * kGallPl] = Qn;
    if (k == kmax) Q[((size_t)p * K + K - 1) * kGallPl] = Qn;
  }
}

// One column per thread and two tracers (an odd group's last one alone): the two share the column's
// density, w and limiter parameters and fill each other's latencies.  The next level's inputs are
// copied to shared memory while a level is worked on, which leaves the registers for three blocks an
// SM: 0.81 ms for 5 tracers at glevel 7, kall 61 (the next level's inputs in registers, two blocks:
// 0.89; one tracer a thread 0.97; a third stage takes the L1 cache away: 1.08).  A column block's
// tracer pairs are consecutive blocks and share rhog, rhogw and the fluxes in L2.
// Level k gives Qout of level k-1 and the limited flux of the face below it, which finish level k-2;
// levels alternate between two slots, so nothing is copied from level to level.
template <int NT>
__device__ __forceinline__ void column(const PlainArgs &P, int t0, int l, int col) {
  const Dims &D = P.D;
  const int n = D.gmax - D.gmin + 1;
  if (col >= n * n) return;
  const int G = D.gall_1d, K = D.kall;
  const unsigned g = (unsigned)D.gall, c = (unsigned)((col / n + D.gmin - 1) * G + col % n + D.gmin - 1);
  const size_t n3 = P.n3(), base = (size_t)l * K * D.gall;
  // addresses: a base that is the same for the whole block, and a 32-bit offset within the region
  const double *flx = P.flx + base, *rho = P.rho + base, *W = P.w + base;
  double *Q[NT];
  const double *fv[NT];
#pragma unroll
  for (int h = 0; h < NT; ++h) Q[h] = P.Q + (size_t)(t0 + h) * n3 + base, fv[h] = P.fv + (size_t)(t0 + h) * 3 * n3 + base;
  // the inputs of kColStages levels, each thread's own copies (cp.async: no barrier, no registers)
  struct In {
    double flx[6], rho, w, x[NT][7];  // x: Q, then the six face values
  };
  constexpr int NV = 8 + 7 * NT;
  extern __shared__ __align__(16) double ring[];  // [stage][value][thread]
  auto issue = [&](int k, bool phys) {
    if (k <= K - 1) {
      double *to = ring + (size_t)(k % kColStages) * NV * kColThreads + threadIdx.x;
      const unsigned o = (unsigned)k * g + c;
#pragma unroll
      for (int m = 0; m < 6; ++m) copy_async(to + m * kColThreads, flx + m * n3 + o);
      copy_async(to + 6 * kColThreads, rho + o), copy_async(to + 7 * kColThreads, W + o);
      if (phys) {
        const unsigned o4 = o - 1, o5 = o - G - 1, o6 = o - G;
#pragma unroll
        for (int h = 0; h < NT; ++h) {
          double *th = to + (8 + 7 * h) * kColThreads;
          copy_async(th, Q[h] + o);
          copy_async(th + kColThreads, fv[h] + o), copy_async(th + 2 * kColThreads, fv[h] + n3 + o);
          copy_async(th + 3 * kColThreads, fv[h] + 2 * n3 + o), copy_async(th + 4 * kColThreads, fv[h] + o4);
          copy_async(th + 5 * kColThreads, fv[h] + n3 + o5), copy_async(th + 6 * kColThreads, fv[h] + 2 * n3 + o6);
        }
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  auto load = [&](In &v, int k) {  // level k, copied kColStages - 1 levels ago
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kColStages - 2) : "memory");
    const double *from = ring + (size_t)(k % kColStages) * NV * kColThreads + threadIdx.x;
#pragma unroll
    for (int m = 0; m < 6; ++m) v.flx[m] = from[m * kColThreads];
    v.rho = from[6 * kColThreads], v.w = from[7 * kColThreads];
#pragma unroll
    for (int h = 0; h < NT; ++h)
#pragma unroll
      for (int m = 0; m < 7; ++m) v.x[h][m] = from[(8 + 7 * h + m) * kColThreads];
  };
  auto horiz = [&](const In &v, int h) {  // rhogq after the horizontal sub-step
    double s = v.flx[0] * v.x[h][1];
#pragma unroll
    for (int m = 1; m < 6; ++m) s = s + v.flx[m] * v.x[h][m + 1];
    return v.x[h][0] - s;
  };
  const int kmin = D.kmin - 1, kmax = D.kmax - 1;
#pragma unroll
  for (int d = 0; d < kColStages - 1; ++d) issue(kmin + d, kmin + d <= kmax);
  if (K == 1) {
    In v;
    load(v, kmin);
#pragma unroll
    for (int h = 0; h < NT; ++h) Q[h][c] = horiz(v, h);
    return;
  }
  // slot s of a window: the level being worked on (before: level k-2); slot 1 - s: level k-1
  double q[NT][2], Qh[NT][2], Qmn[NT], Qmx[NT], fl[NT];
  double c1 = 0.0, wk = 0.0;  // ck1 and w of level k-1
  Recip rp{1.0, 1.0, true};   // its density
  auto level = [&](int k, auto slot) {
    constexpr int S = decltype(slot)::value, Z = 1 - S;
    In v;
    load(v, k);
    issue(k + kColStages - 1, k + kColStages - 1 <= kmax);  // into the stage of level k - 1
    double r = v.flx[0];
#pragma unroll
    for (int m = 1; m < 6; ++m) r = r + v.flx[m];
    const Recip rr = recip(v.rho - r);
    double x[1 + NT] = {-v.w * P.dt * P.rdgz[k]}, Qn[NT] = {};  // ck1, q of the tracers
    if (k <= kmax) {
#pragma unroll
      for (int h = 0; h < NT; ++h) x[1 + h] = Qn[h] = horiz(v, h);
    }
    quotients(x, rr);
    if (k == kmin) {
#pragma unroll
      for (int h = 0; h < NT; ++h) {
        Qh[h][S] = Qn[h], q[h][S] = q[h][Z] = x[1 + h];
        Qmn[h] = Qmx[h] = fl[h] = 0.0;
      }
    } else {
      double c2[1] = {v.w * P.dt * P.rdgz[k - 1]};  // ck2 of level k-1
      quotients(c2, rp);
      const VPar vp = vpar(c1, c2[0], x[0]);
      const double af = P.afact[k - 1], bf = P.bfact[k - 1];
#pragma unroll
      for (int h = 0; h < NT; ++h) {
        const double qn = k <= kmax ? x[1 + h] : q[h][Z];  // the ghost above repeats the top level
        double lo, hi;
        vqout(vp, q[h][S], q[h][Z], qn, lo, hi);
        double qh = af * q[h][Z] + bf * q[h][S];
        if (k - 1 > kmin) qh = vclamp(vp.infl, qh, Qmn[h], Qmx[h], lo, hi);
        const double fu = wk * qh;  // through the face below level k-1
        if (k - 1 > kmin) {
          const double z = Qh[h][S] - (fu - fl[h]) * P.dt * P.rdgz[k - 2];
          Q[h][(unsigned)(k - 2) * g + c] = z;
          if (k - 2 == kmin) Q[h][c] = z;
        }
        fl[h] = fu, Qmn[h] = lo, Qmx[h] = hi;
        Qh[h][S] = Qn[h], q[h][S] = qn;
      }
    }
    c1 = x[0], rp = rr, wk = v.w;
  };
  using C0 = std::integral_constant<int, 0>;
  using C1 = std::integral_constant<int, 1>;
  auto top = [&](auto slot) {  // level kmax: the flux through the top face is unlimited
    constexpr int S = decltype(slot)::value, Z = 1 - S;  // S: the ghost level's slot, Z: kmax's
#pragma unroll
    for (int h = 0; h < NT; ++h) {
      const double qh = P.afact[kmax + 1] * q[h][S] + P.bfact[kmax + 1] * q[h][Z];
      const double z = Qh[h][Z] - (wk * qh - fl[h]) * P.dt * P.rdgz[kmax];
      Q[h][(unsigned)kmax * g + c] = z;
      Q[h][(unsigned)(K - 1) * g + c] = z;
      if (kmin == kmax) Q[h][c] = z;
    }
  };
#pragma unroll 1
  for (int k = kmin;; k += 2) {
    level(k, C0{});
    if (k == kmax + 1) {
      top(C0{});
      break;
    }
    level(k + 1, C1{});
    if (k + 1 == kmax + 1) {
      top(C1{});
      break;
    }
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// blocks: (tracer pair fastest, column block, region), then the pole columns
__global__ void __launch_bounds__(kColThreads, kColBlocks) k_plain_column(PlainArgs P, int colblk, int nmain) {
  if ((int)blockIdx.x >= nmain) {
    const int u = (int)blockIdx.x - nmain;
    pole_column(P, u % kLallPl, u / kLallPl);
    return;
  }
  const int npair = (P.nt + 1) / 2, t0 = (int)blockIdx.x % npair * 2, cb = (int)blockIdx.x / npair;
  const int l = cb / colblk, col = cb % colblk * kColThreads + (int)threadIdx.x;
  if (t0 + 1 < P.nt) column<2>(P, t0, l, col);
  else column<1>(P, t0, l, col);
}

// the density: rhog -= sum_m flx_h(m), then -= d(rhogw)/dz dt, ghost levels copied.  One thread per
// (cell, level), after every tracer has read the old density; the last threads take the pole centres.
__global__ void k_plain_rho(Dims D, double dt, const double *flx, const double *flx_pl, const double *w,
                            const double *w_pl, const double *rdgz, double *rho, double *rho_pl) {
  const int n = D.gmax - D.gmin + 1, K = D.kall, kmin = D.kmin - 1, kmax = D.kmax - 1, NK = kmax - kmin + 1;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, nc = (long long)D.lall * NK * n * n;
  double *R, *col;
  const double *W;
  double s;
  size_t lev;
  int k;
  if (t < nc) {
    const int r = (int)(t % (n * n)), c = (r / n + D.gmin - 1) * D.gall_1d + r % n + D.gmin - 1;
    k = kmin + (int)(t / (n * n) % NK);
    const size_t n3 = (size_t)D.lall * K * D.gall, cb = (size_t)(t / (n * n) / NK) * K * D.gall + c;
    lev = D.gall;
    const size_t o = cb + k * lev;
    col = rho + cb, R = rho + o, W = w + o;
    s = flx[o];
    for (int m = 1; m < 6; ++m) s = s + flx[m * n3 + o];
  } else if (t < nc + kLallPl * NK) {
    const int p = (int)(t - nc) / NK;
    k = kmin + (int)(t - nc) % NK;
    lev = kGallPl;
    const size_t cb = (size_t)p * K * kGallPl, o = cb + k * lev;
    col = rho_pl + cb, R = rho_pl + o, W = w_pl + o;
    s = flx_pl[o + 1];
    for (int v = 2; v <= 5; ++v) s = s + flx_pl[o + v];
  } else {
    return;
  }
  double r = *R - s;
  if (K > 1) r = r - (W[lev] - W[0]) * dt * rdgz[k];
  *R = r;
  if (k == kmin && k != 0) col[0] = r;
  if (k == kmax && k != K - 1) col[(size_t)(K - 1) * lev] = r;
}

// ---------------------------------------------------------------------------
static size_t n3_of(const Dims &D) { return (size_t)D.gall * D.kall * D.lall; }
static size_t n3p_of(const Dims &D) { return (size_t)kGallPl * D.kall * kLallPl; }

template <int TX>
static cudaError_t launch_cells(const PlainArgs &P, cudaStream_t st) {
  const Dims &D = P.D;
  using S = typename CellTile<TX, kTileCells>::Smem;
  const int n = D.gmax - D.gmin + 1, ntx = (n + TX - 1) / TX, nty = (n + S::TY - 1) / S::TY;
  const int tiles = ntx * nty * D.lall, NK = D.kmax - D.kmin + 1;
  // up to 8 levels a block (the gradient coefficients are loaded once per block), fewer while
  // that leaves less than two waves of the 2 blocks an SM holds
  int lpb = 8;
  while (lpb > 1 && (long long)tiles * ((NK + lpb - 1) / lpb) < 2 * 2 * 148) lpb /= 2;
  const int nlb = (NK + lpb - 1) / lpb;
  const int npole = (P.nt * kLallPl * D.kall + kTileCells - 1) / kTileCells;
  cudaError_t e = cudaFuncSetAttribute(k_plain_cells<TX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(S));
  if (e != cudaSuccess) return e;
  k_plain_cells<TX><<<(unsigned)(tiles * nlb + npole), kTileCells, sizeof(S), st>>>(P, ntx, nty, nlb, lpb);
  return cudaGetLastError();
}

PlainArgs plain_group(const StepCtx &S, int t0, int ntr, double dt, const double *rhog, const double *rhog_pl,
                      double *rhogq, double *rhogq_pl, const double *w, const double *w_pl) {
  const Dims &D = S.D;
  PlainArgs P{};
  P.D = D, P.nt = (ntr - t0 < kPlainGroup) ? ntr - t0 : kPlainGroup, P.nb = S.nb, P.ns = S.ns, P.dt = dt;
  P.Q = rhogq + t0 * n3_of(D), P.Qp = rhogq_pl + t0 * n3p_of(D);
  P.rho = rhog, P.rhop = rhog_pl, P.w = w, P.wp = w_pl;
  P.flx = S.flx, P.flxp = S.flx_pl, P.xc = S.xc, P.xcp = S.xc_pl;
  P.GRD_x = S.GRD_x, P.GRD_xp = S.GRD_x_pl, P.cg = S.cg, P.cgp = S.cg_pl;
  P.rdgz = S.rdgz, P.afact = S.afact, P.bfact = S.bfact;
  P.bsrc = S.bsrc, P.seam = S.seam, P.ring = S.ring;
  P.fv = S.fv, P.bb = S.bb;
  return P;
}

int plain_faces(const PlainArgs &P, cudaStream_t st, long long &launches) {
  const int n = P.D.gmax - P.D.gmin + 1, NK = P.D.kmax - P.D.kmin + 1;
  // 32 x 8 tiles need no partial tile in any region 32 or more cells wide (a region is a power of two wide)
  const cudaError_t e = n >= 32 ? launch_cells<32>(P, st) : launch_cells<16>(P, st);
  if (e != cudaSuccess) return set_error(std::string("advect_step: ") + cudaGetErrorString(e)), ICA_ERR_CUDA;
  const long long ns = (long long)P.ns * NK;
  k_plain_seam<<<(unsigned)((ns + 127) / 128), 128, 0, st>>>(P);
  launches += 2;
  return ICA_OK;
}

int step_plain(StepCtx &S, int ntr, double dt, double *rhog, double *rhog_pl, double *rhogq, double *rhogq_pl,
               const double *vx, const double *vx_pl, const double *vy, const double *vy_pl, const double *vz,
               const double *vz_pl, const double *w, const double *w_pl, cudaStream_t st, long long &launches) {
  const Dims &D = S.D;
  if (D.kall > kColThreads) return set_error("advect_step: kall above 128"), ICA_ERR_ARG;
  FluxIn<double> fin{rhog, rhog_pl, vx, vx_pl, vy, vy_pl, vz, vz_pl};
  FluxOut<double> fout{S.flx, S.flx_pl, S.xc, S.xc_pl};
  launch_horizontal_flux<double>(D, fin, fout, S.geo, dt, st);
  launches += 1;
  const int n = D.gmax - D.gmin + 1, NK = D.kmax - D.kmin + 1;
  const int colblk = (n * n + kColThreads - 1) / kColThreads;  // column blocks of a region
  const cudaError_t e = cudaFuncSetAttribute(k_plain_column, cudaFuncAttributeMaxDynamicSharedMemorySize, kColSmem);
  if (e != cudaSuccess) return set_error(std::string("advect_step: ") + cudaGetErrorString(e)), ICA_ERR_CUDA;
  for (int t0 = 0; t0 < ntr; t0 += kPlainGroup) {
    const PlainArgs P = plain_group(S, t0, ntr, dt, rhog, rhog_pl, rhogq, rhogq_pl, w, w_pl);
    const int rc = plain_faces(P, st, launches);
    if (rc) return rc;
    const int nmain = colblk * D.lall * ((P.nt + 1) / 2);
    k_plain_column<<<(unsigned)(nmain + kLallPl * P.nt), kColThreads, kColSmem, st>>>(P, colblk, nmain);
    launches += 1;
  }
  const long long nr = ((long long)D.lall * n * n + kLallPl) * NK;
  k_plain_rho<<<(unsigned)((nr + 255) / 256), 256, 0, st>>>(D, dt, S.flx, S.flx_pl, w, w_pl, S.rdgz, rhog, rhog_pl);
  launch_gather<double>(D, S.plan.n, S.plan.dst, S.plan.src, D.kall, ntr, rhogq, rhogq_pl, st, rhog, rhog_pl);
  launches += 2;
  return ICA_OK;
}

}  // namespace icoadv
