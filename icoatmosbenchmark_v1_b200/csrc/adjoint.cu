// Reverse mode (adjoint) of the composed FP64 step of step.cu.
//
// Given the step's input state (a checkpoint) and the adjoint of its output,
// the forward intermediates are recomputed with the step's own kernels, then
// every operation is transposed in reverse order: the final halo fill, the
// vertical sub-step (column by column), the horizontal rhogq update, the
// limiter apply and the Qout halo fill, the Qout bounds, the upwind remap,
// the gradient and its halo fill, q = rhogq / rhog, the density update, the
// Courant numbers and horizontal_flux (dyn_horiz_adv_flux/src/
// mod_src_tracer.f90:42-379), whose triangle interpolation carries the
// adjoint to rhog and the three wind components.
//
// Kinks follow the forward's own comparisons (subgradients, as in
// tangent-linear models): min/max pass the adjoint to the operand the forward
// returned (the first one on a tie), a clamp to its input when the input was
// returned and to the binding bound otherwise; the upwind masks, inflow flags
// and zero-outflow switches are held fixed; terms that carry +-BIG (the
// outflow side of a masked bound) have no derivative.  rhogw, the geometry
// and the vertical grid are constants.
//
// The horizontal sub-step is transposed where the forward forms it: by the thread of a
// face's upwind cell, which holds every operand (k_adj_cells), with the seam faces in
// a kernel of their own.  What the data decide (a bound handing its adjoint to one of
// its cells, a halo copy to its source) and sums over tiles and tracers use FP64
// atomicAdd; the triangle interpolation is transposed as a gather.  Sums therefore
// associate differently from a serial adjoint, at rounding level.
#include <cuda_runtime.h>

#include <cfloat>

#include "adjoint.cuh"
#include "plain_cells.cuh"

namespace icoadv {

namespace {

constexpr double kEps = DBL_EPSILON, kBig = DBL_MAX;

__device__ __forceinline__ bool inner(const Dims &D, int i, int j) {
  return i >= D.gmin && i <= D.gmax && j >= D.gmin && j <= D.gmax;
}

// The arguments of a group of tracers.
struct AdjArgs {
  PlainArgs P;
  double *aQ, *aQp;      // the group's adjoint of rhogq
  double *Qh, *Qhp;      // rhogq after the horizontal sub-step (Qh: a_q's memory, until the column pass is done)
  double *a_q, *a_qp;    // adjoint of q
  double *a_bb;          // adjoint of the boundary values: gradient x/y/z, Qout min / max
  double *rh, *rhp, *a_rh, *a_rhp, *a_flx, *a_flxp, *a_xc, *a_xcp, *a_chp, *a_rho, *a_rhop;
  bool first, last;      // of the step's groups
  __device__ double *abval(int t, int k, int b) const { return a_bb + (((size_t)t * P.D.kall + k) * P.nb + b) * 5; }
};

// Limiter apply and remap of a face's value v0 (bounds lo, hi; the upwind cell's Qout Qn, Qx): the
// limited value, and what it is a copy of (mod_src_tracer.f90:378-410).
enum Pick { kRemap, kLow, kHigh, kQmin, kQmax };
__device__ __forceinline__ Pick limited(double v0, double lo, double hi, double Qn, double Qx) {
  const double v1a = mx(v0, lo), v1 = mn(v1a, hi), v2a = mn(v1, Qx);
  if (Qn > v2a) return kQmin;
  if (Qx < v1) return kQmax;
  if (hi < v1a) return kHigh;
  return (lo > v0) ? kLow : kRemap;
}

// ---------------------------------------------------------------------------
// halo fill: every copied point hands its adjoint to its source and drops it
// (the composed plan never reads a point it writes)
__global__ void k_fill_adj(int nent, const int *__restrict__ dst, const int *__restrict__ src, int npt_rgn,
                           int gall, int lall, int kmax, int vmax, double *a, double *a_pl) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)nent * kmax * vmax) return;
  const int e = (int)(t % nent), kv = (int)(t / nent), k = kv % kmax, v = kv / kmax;
  auto addr = [&](int p) -> double * {
    if (p < npt_rgn) return a + (((size_t)v * lall + p / gall) * kmax + k) * gall + p % gall;
    const int qd = p - npt_rgn;
    return a_pl + (((size_t)v * kLallPl + qd / kGallPl) * kmax + k) * kGallPl + qd % kGallPl;
  };
  double *pd = addr(dst[e]);
  const double x = *pd;
  if (x == 0.0) return;
  *pd = 0.0;
  atomicAdd(addr(src[e]), x);
}

// ---------------------------------------------------------------------------
// vertical sub-step, density part: rhog(kall) = rhog(kmax), rhog(1) = rhog(kmin),
// rhog(k) = rho_h(k) - d(rhogw)/dz dt.  The adjoint of rho_h goes to a_rh; the
// input adjoint (a_rho in place) keeps what passes through the step unchanged
// (halo columns, pole ring points) and is zero elsewhere so far.
__global__ void k_adj_vrho(Dims D, double *a_rho, double *a_rho_pl, double *a_rh, double *a_rh_pl) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int ncol = D.lall * D.gall;
  double *aR, *aH;
  size_t s;
  bool col;
  if (t < ncol) {
    const int l = t / D.gall, c = t % D.gall, G = D.gall_1d;
    const size_t base = (size_t)l * D.kall * D.gall + c;
    aR = a_rho + base, aH = a_rh + base, s = D.gall;
    col = inner(D, c % G + 1, c / G + 1);
  } else if (t < ncol + kLallPl * kGallPl) {
    const int p = t - ncol, l = p / kGallPl, v = p % kGallPl;
    const size_t base = (size_t)l * D.kall * kGallPl + v;
    aR = a_rho_pl + base, aH = a_rh_pl + base, s = kGallPl;
    col = (v == 0);
  } else {
    return;
  }
  const int K = D.kall, kmin = D.kmin - 1, kmax = D.kmax - 1;  // 0-based
  if (!col) {
    for (int k = 0; k < K; ++k) aH[k * s] = 0.0;
    return;
  }
  aR[kmax * s] += aR[(K - 1) * s];
  aR[(K - 1) * s] = 0.0;
  aR[kmin * s] += aR[0];
  aR[0] = 0.0;
  for (int k = 0; k < K; ++k) {
    aH[k * s] = (k >= kmin && k <= kmax) ? aR[k * s] : 0.0;
    aR[k * s] = 0.0;
  }
}

// ---------------------------------------------------------------------------
// vertical sub-step of one tracer, one column per thread, levels streamed from the top.
//
// Forward (step.cu k_plain_column, mod_src_tracer.f90:107-186 with d = 0):
//   qc(k) = Qh(k) / rh(k), ghosts qc(1) = qc(kmin), qc(kall) = qc(kmax)
//   ck1(k) = -w(k) dt rdgz(k) / rh(k), ck2(k) = w(k+1) dt rdgz(k) / rh(k), ck1(kall) likewise
//   qh(k) = afact(k) qc(k) + bfact(k) qc(k-1), clamped to the Qout bounds of level k-1 or k
//   Q(k) = Qh(k) - (w(k+1) qh(k+1) - w(k) qh(k)) dt rdgz(k), ghosts copied
// The column adjoint's per-level inputs stream through a shared-memory ring of kAdjStages
// levels, filled by each thread's own cp.async copies (no barrier: a thread reads only what it
// copied), so kAdjStages - 1 levels of a column are in flight while a level is worked on
// (a 4-step sweep at gl7, 4 tracers: 124.2 -> 118.5 ms against plain loads of each level).
constexpr int kAdjStages = 4, kAdjThreads = 128;
struct AdjRing {
  double v[kAdjStages][6][kAdjThreads];  // Qh(kk), rh(kk), rh(k), w(k), w(k+1), aQ(k)
};
__device__ __forceinline__ unsigned adj_smem_u32(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void adj_cp8(double *dst, const double *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(adj_smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void adj_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void adj_drain() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void adj_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

struct VLev {  // one level's inputs
  double qc, R, w, c1, c2, aO;
};
struct VLim {  // one level's Thuburn bounds and what they were made of
  double infL, infU, c1, c2, mnL, mnU, mxL, mxU, qnmin, qnmax, Cin, Cout, zsw, Qmn, Qmx;
  int amin, amax;
};

__device__ __forceinline__ VLim vlim_level(double qm, double qk, double qp, double c1, double c1u, double c2) {
  VLim v;
  v.infL = 0.5 - sgn(0.5, c1);
  v.infU = 0.5 + sgn(0.5, c1u);
  v.c1 = c1, v.c2 = c2;
  v.mnL = mn(qk, qm) + (1.0 - v.infL) * kBig;
  v.mnU = mn(qk, qp) + (1.0 - v.infU) * kBig;
  v.mxL = mx(qk, qm) - (1.0 - v.infL) * kBig;
  v.mxU = mx(qk, qp) - (1.0 - v.infU) * kBig;
  const double t1 = mn(v.mnL, v.mnU);
  v.qnmin = mn(t1, qk);
  v.amin = (qk < t1) ? 2 : ((v.mnU < v.mnL) ? 1 : 0);
  const double t2 = mx(v.mxL, v.mxU);
  v.qnmax = mx(t2, qk);
  v.amax = (qk > t2) ? 2 : ((v.mxU > v.mxL) ? 1 : 0);
  v.Cin = v.infL * c1 + v.infU * c2;
  v.Cout = (1.0 - v.infL) * c1 + (1.0 - v.infU) * c2;
  const double CQmin = v.infL * c1 * v.mnL + v.infU * c2 * v.mnU;
  const double CQmax = v.infL * c1 * v.mxL + v.infU * c2 * v.mxU;
  v.zsw = 0.5 - sgn(0.5, fabs(v.Cout) - kEps);
  v.Qmn = ((qk - v.qnmax) + v.qnmax * (v.Cin + v.Cout) - CQmax) / (v.Cout + v.zsw) * (1.0 - v.zsw) + qk * v.zsw;
  v.Qmx = ((qk - v.qnmin) + v.qnmin * (v.Cin + v.Cout) - CQmin) / (v.Cout + v.zsw) * (1.0 - v.zsw) + qk * v.zsw;
  return v;
}

// adjoint of (Qout_min, Qout_max) of one level -> qc(k-1), qc(k), qc(k+1), ck1(k), ck2(k)
__device__ __forceinline__ void vlim_level_adj(const VLim &v, double qm, double qk, double qp, double aQm,
                                               double aQx, double &am, double &a0, double &ap, double &ac1,
                                               double &ac2) {
  if (aQm == 0.0 && aQx == 0.0) return;
  if (v.zsw != 0.0) {
    a0 += aQm + aQx;
    return;
  }
  const double c1 = v.c1, c2 = v.c2;
  const double Dn = v.Cout, S = v.Cin + v.Cout;
  const double CQmax = v.infL * c1 * v.mxL + v.infU * c2 * v.mxU;
  const double CQmin = v.infL * c1 * v.mnL + v.infU * c2 * v.mnU;
  const double Nmn = (qk - v.qnmax) + v.qnmax * S - CQmax, Nmx = (qk - v.qnmin) + v.qnmin * S - CQmin;
  const double rD = 1.0 / Dn;
  const double aNmn = aQm * rD, aNmx = aQx * rD;
  const double aD = -(aNmn * Nmn + aNmx * Nmx) * rD;
  double a_qk = aNmn + aNmx;
  const double a_qnmax = aNmn * (S - 1.0), a_qnmin = aNmx * (S - 1.0);
  const double aS = aNmn * v.qnmax + aNmx * v.qnmin;
  const double aCQmax = -aNmn, aCQmin = -aNmx;
  const double aCin = aS, aCout = aS + aD;
  double amxL = aCQmax * v.infL * c1, amxU = aCQmax * v.infU * c2;
  double amnL = aCQmin * v.infL * c1, amnU = aCQmin * v.infU * c2;
  double a1 = aCin * v.infL + aCout * (1.0 - v.infL);
  double a2 = aCin * v.infU + aCout * (1.0 - v.infU);
  if (v.infL != 0.0) a1 += aCQmax * v.infL * v.mxL + aCQmin * v.infL * v.mnL;
  if (v.infU != 0.0) a2 += aCQmax * v.infU * v.mxU + aCQmin * v.infU * v.mnU;
  if (v.amax == 2) a_qk += a_qnmax;
  else if (v.amax == 1) amxU += a_qnmax;
  else amxL += a_qnmax;
  if (v.amin == 2) a_qk += a_qnmin;
  else if (v.amin == 1) amnU += a_qnmin;
  else amnL += a_qnmin;
  if (v.infL != 0.0) {
    if (qm < qk) am += amnL;
    else a_qk += amnL;
    if (qm > qk) am += amxL;
    else a_qk += amxL;
  }
  if (v.infU != 0.0) {
    if (qp < qk) ap += amnU;
    else a_qk += amnU;
    if (qp > qk) ap += amxU;
    else a_qk += amxU;
  }
  a0 += a_qk;
  ac1 += a1;
  ac2 += a2;
}

// Blocks: tracers fastest (they share rh and w in L2), column blocks of a region, regions; the last
// blocks take the pole columns.
__global__ void __launch_bounds__(kAdjThreads) k_adj_vert(AdjArgs A, int colblk, int nmain) {
  const Dims &D = A.P.D;
  const double dt = A.P.dt, *__restrict__ rdgz = A.P.rdgz, *__restrict__ afact = A.P.afact, *__restrict__ bfact = A.P.bfact;
  const double *QH, *R, *W;
  double *AQ, *ARH;
  size_t s;
  if ((int)blockIdx.x < nmain) {
    const int t = (int)blockIdx.x % A.P.nt, cb = (int)blockIdx.x / A.P.nt, l = cb / colblk;
    const int n = D.gmax - D.gmin + 1, col = cb % colblk * kAdjThreads + (int)threadIdx.x;
    if (col >= n * n) return;
    const size_t base = (size_t)l * D.kall * D.gall + (col / n + D.gmin - 1) * D.gall_1d + col % n + D.gmin - 1;
    const size_t tb = t * A.P.n3() + base;
    QH = A.Qh + tb, R = A.rh + base, W = A.P.w + base, AQ = A.aQ + tb, ARH = A.a_rh + base, s = D.gall;
  } else {
    const int u = ((int)blockIdx.x - nmain) * kAdjThreads + (int)threadIdx.x;
    if (u >= kLallPl * A.P.nt) return;
    const size_t base = (size_t)(u % kLallPl) * D.kall * kGallPl, tb = u / kLallPl * A.P.n3p() + base;
    QH = A.Qhp + tb, R = A.rhp + base, W = A.P.wp + base, AQ = A.aQp + tb, ARH = A.a_rhp + base, s = kGallPl;
  }
  const int K = D.kall, kmin = D.kmin, kmax = D.kmax;  // 1-based levels below
  auto X = [&](int k) { return (size_t)(k - 1) * s; };
  const double aTop = AQ[X(K)], aBot = AQ[X(1)];
  extern __shared__ __align__(16) unsigned char adj_raw[];
  AdjRing &ring = *reinterpret_cast<AdjRing *>(adj_raw);
  const int th = threadIdx.x;
  // the levels are taken in the order K, K-1, ..., 1: level j's inputs into slot j % kAdjStages
  auto issue = [&](int j) {
    if (j >= 1) {
      const int sl = j % kAdjStages, kk = (j < kmin) ? kmin : ((j > kmax) ? kmax : j);
      adj_cp8(&ring.v[sl][0][th], QH + X(kk));
      adj_cp8(&ring.v[sl][1][th], R + X(kk));
      adj_cp8(&ring.v[sl][2][th], R + X(j));
      adj_cp8(&ring.v[sl][3][th], W + X(j));
      adj_cp8(&ring.v[sl][4][th], W + X(j < K ? j + 1 : K));
      adj_cp8(&ring.v[sl][5][th], AQ + X(j));
    }
    adj_commit();
  };
#pragma unroll
  for (int d = 0; d < kAdjStages - 1; ++d) issue(K - d);
  auto level = [&](int k) {
    adj_wait<kAdjStages - 2>();  // level k's copies are complete
    const int sl = k % kAdjStages;
    const double vq = ring.v[sl][0][th], vrk = ring.v[sl][1][th], vr = ring.v[sl][2][th];
    const double vw = ring.v[sl][3][th], vw1 = ring.v[sl][4][th], va = ring.v[sl][5][th];
    issue(k - (kAdjStages - 1));  // into the slot of level k + 1, read in the previous call
    VLev v;
    v.qc = vq / vrk;
    v.R = vr;
    v.w = vw;
    v.c1 = v.c2 = v.aO = 0.0;
    if (k >= kmin && k <= kmax) {
      v.c1 = -v.w * dt * rdgz[k - 1] / v.R;
      v.c2 = vw1 * dt * rdgz[k - 1] / v.R;
      double a = va;
      if (k == kmax) a = a + aTop;
      if (k == kmin) a = a + aBot;
      v.aO = a;
    } else if (k == K) {
      v.c1 = -v.w * dt * rdgz[k - 1] / v.R;
    }
    return v;
  };
  // window: levels k+1 (P), k (Z), k-1 (M), k-2 (M2); the Thuburn bounds of a level are
  // recomputed where they are needed instead of carried, which keeps the thread's state small
  VLev P{}, Z = level(K), M = level(K - 1), M2{};
  double aQmZ = 0.0, aQxZ = 0.0, aQmM = 0.0, aQxM = 0.0;  // adjoints of the Qout bounds of k, k-1
  double accP = 0.0, accZ = 0.0, accM = 0.0;             // limiter adjoints into qc(k+1), qc(k), qc(k-1)
  double ac1P = 0.0, ac2P = 0.0;                          // adjoints of ck1, ck2 of level k+1
  double ahP2 = 0.0, ahP = 0.0;                           // post-clamp adjoints of qh(k+2), qh(k+1)
  double aqcTop = 0.0;                                    // adjoint of the ghost qc(kall)
  for (int k = K; k >= kmin; --k) {
    if (k - 2 >= 1) M2 = level(k - 2);
    // qh(k) from the rhogq update of levels k-1 and k
    double ah;
    {
      const bool lo = (k - 1 >= kmin), hi = (k <= kmax);
      const double t1 = lo ? -M.aO * Z.w * dt * rdgz[k - 2] : 0.0;
      const double t2 = hi ? Z.aO * Z.w * dt * rdgz[k - 1] : 0.0;
      ah = (lo && hi) ? t1 + t2 : (lo ? t1 : t2);
    }
    double ac1Z = 0.0, ac2Z = 0.0;
    if (k <= kmax) {
      const VLim LZ = vlim_level(M.qc, Z.qc, P.qc, Z.c1, P.c1, Z.c2);
      // the clamp of qh(k) to the bounds of level k-1 (inflow from below) or k
      if (k >= kmin + 1) {
        const bool below = (LZ.infL != 0.0);
        double Qmx = LZ.Qmx, Qmn = LZ.Qmn;
        if (below) {
          const VLim LM = vlim_level(M2.qc, M.qc, Z.qc, M.c1, Z.c1, M.c2);
          Qmx = LM.Qmx, Qmn = LM.Qmn;
        }
        const double h = afact[k - 1] * Z.qc + bfact[k - 1] * M.qc;
        const double m1 = mn(h, Qmx);
        int sel = (Qmx < h) ? 1 : 0;
        if (Qmn > m1) sel = 2;
        if (sel == 1) {
          if (below) aQxM += ah;
          else aQxZ += ah;
          ah = 0.0;
        } else if (sel == 2) {
          if (below) aQmM += ah;
          else aQmZ += ah;
          ah = 0.0;
        }
      }
      // Qout bounds of level k
      vlim_level_adj(LZ, M.qc, Z.qc, P.qc, aQmZ, aQxZ, accM, accZ, accP, ac1Z, ac2Z);
    }
    // level k+1 is complete
    if (k + 1 == K) {
      aqcTop = accP + afact[K - 1] * ahP;
    } else if (k + 1 <= kmax) {
      double a = accP;
      a += afact[k] * ahP;
      a += bfact[k + 1] * ahP2;
      if (k + 1 == kmax) a += aqcTop;
      const double rR = 1.0 / P.R;
      AQ[X(k + 1)] = P.aO + a * rR;
      atomicAdd(&ARH[X(k + 1)], -a * P.qc * rR - (ac1P * P.c1 + ac2P * P.c2) * rR);  // the tracers share rh
    }
    // shift the window down one level
    P = Z, Z = M, M = M2;
    aQmZ = aQmM, aQxZ = aQxM, aQmM = aQxM = 0.0;
    accP = accZ, accZ = accM, accM = 0.0;
    ac1P = ac1Z, ac2P = ac2Z;
    ahP2 = ahP, ahP = ah;
  }
  // level kmin (now P) with the ghost qc(1) (now Z's accumulator)
  {
    const double aqcBot = accZ + bfact[kmin - 1] * ahP;
    double a = accP;
    a += afact[kmin - 1] * ahP;
    a += bfact[kmin] * ahP2;
    if (kmin == kmax) a += aqcTop;
    a += aqcBot;
    const double rR = 1.0 / P.R;
    AQ[X(kmin)] = P.aO + a * rR;
    atomicAdd(&ARH[X(kmin)], -a * P.qc * rR - (ac1P * P.c1 + ac2P * P.c2) * rR);
  }
  AQ[X(1)] = 0.0;
  AQ[X(K)] = 0.0;
  adj_drain();
}

// ---------------------------------------------------------------------------
// The horizontal sub-step.  The forward's own kernels (plain_faces) recompute every limited face value
// fv and the boundary values bb; the gradient, bounds and Qout of a cell are formed again where they
// are transposed, from q in shared memory as the forward forms them, and never stored.

// One of the five faces of pole p at level k (v = 1..5: ring slot), tracer t: forward values.
struct PoleFace {
  double q[kGallPl], lo, hi, v0;
  int up;            // the upwind point's slot, 0: the centre
  const double *bv;  // its gradient and Qout
};
__device__ __forceinline__ PoleFace pole_face(const PlainArgs &P, int t, int p, int k, int v) {
  const size_t off = ((size_t)p * P.D.kall + k) * kGallPl, n3p = P.n3p();
  PoleFace f;
#pragma unroll
  for (int x = 0; x < kGallPl; ++x) f.q[x] = P.Qp[t * n3p + off + x] / P.rhop[off + x];
  const int vp = (v == 5) ? 1 : v + 1, vm = (v == 1) ? 5 : v - 1;
  auto q = [&](int x) { return P.Qp[t * n3p + off + x] / P.rhop[off + x]; };
  const double qv = q(v), qm = q(vm), qp = q(vp);
  f.up = upmask(P.flxp[off + v], P.rhop[off]) ? v : 0;
  f.bv = P.bval(t, k, f.up ? P.ring[p * kVlink + v - 1] : P.nb - 2 + p);
  f.lo = mn4(f.q[0], qv, qm, qp), f.hi = mx4(f.q[0], qv, qm, qp);
  f.v0 = f.up ? qv : f.q[0];
  for (int d = 0; d < 3; ++d)
    f.v0 = f.v0 + f.bv[d] * (P.xcp[d * n3p + off + v] - P.GRD_xp[((size_t)d * kLallPl + p) * kGallPl + f.up]);
  return f;
}

// rhogq after the horizontal sub-step from the face values (one thread per cell and level, the
// group's tracers one after the other), and with the first group the density after it.  The last
// blocks take the pole centres.
__global__ void __launch_bounds__(128) k_adj_qh(AdjArgs A, int cellblk, int nmain) {
  const PlainArgs &P = A.P;
  const Dims &D = P.D;
  const size_t n3 = P.n3(), n3p = P.n3p();
  const int K = D.kall;
  if ((int)blockIdx.x >= nmain) {
    const int u = ((int)blockIdx.x - nmain) * 128 + (int)threadIdx.x;
    if (u >= P.nt * kLallPl * K) return;
    const int k = u % K, p = u / K % kLallPl, t = u / K / kLallPl;
    const size_t off = ((size_t)p * K + k) * kGallPl;
    double s = 0.0, r = 0.0;
    for (int v = 1; v <= 5; ++v) {
      const double f = P.flxp[off + v];
      r = (v == 1) ? f : r + f;
      if (k >= D.kmin - 1 && k < D.kmax) {
        const PoleFace F = pole_face(P, t, p, k, v);
        const double x = mx(mn(mn(mx(F.v0, F.lo), F.hi), F.bv[4]), F.bv[3]);
        s = (v == 1) ? f * x : s + f * x;
      }
    }
    A.Qhp[t * n3p + off] = P.Qp[t * n3p + off] - s;
    if (t == 0) A.rhp[off] = P.rhop[off] - r;
    return;
  }
  const int ci = (int)blockIdx.x % cellblk * 128 + (int)threadIdx.x, kl = (int)blockIdx.x / cellblk, k = kl % K;
  const int G = D.gall_1d;
  if (ci >= D.gall || !inner(D, ci % G + 1, ci / G + 1)) return;
  const unsigned c = ci;
  const size_t off = (size_t)kl * D.gall;
  double f[6];
#pragma unroll
  for (int m = 0; m < 6; ++m) f[m] = (P.flx + m * n3 + off)[c];
  if (A.first) A.rh[off + c] = P.rho[off + c] - (f[0] + f[1] + f[2] + f[3] + f[4] + f[5]);
  if (k < D.kmin - 1 || k >= D.kmax) return;
  for (int t = 0; t < P.nt; ++t) {
    const double *fv = P.fv + (size_t)t * 3 * n3 + off;
    double s = f[0] * fv[c];
    s = s + f[1] * (fv + n3)[c];
    s = s + f[2] * (fv + 2 * n3)[c];
    s = s + f[3] * fv[c - 1];
    s = s + f[4] * (fv + n3)[c - G - 1];
    s = s + f[5] * (fv + 2 * n3)[c - G];
    (A.Qh + t * n3 + off)[c] = (P.Q + t * n3 + off)[c] - s;
  }
}

// which of four values mn4 / mx4 returns
__device__ __forceinline__ int arg4(const double (&v)[4], bool high) {
  int i = 0;
  double s = v[0];
#pragma unroll
  for (int n = 1; n < 4; ++n)
    if (high ? v[n] > s : v[n] < s) s = v[n], i = n;
  return i;
}

// Faces with a halo cell on one side, one thread per (face, level), the group's tracers one after the
// other: the adjoint of the upwind cell's gradient and Qout goes to the cell whose values the halo
// stands for (a_bb).  The last threads take the pole faces.
__global__ void __launch_bounds__(128) k_adj_seam(AdjArgs A) {
  const PlainArgs &P = A.P;
  const Dims &D = P.D;
  const int NK = D.kmax - D.kmin + 1, K = D.kall, G = D.gall_1d;
  const size_t n3 = P.n3(), n3p = P.n3p();
  const long long u = (long long)blockIdx.x * 128 + threadIdx.x, nseam = (long long)P.ns * NK;
  if (u >= nseam) {
    const int w = (int)(u - nseam);
    if (w >= kLallPl * NK * 5 * P.nt) return;
    const int v = w % 5 + 1, k = D.kmin - 1 + w / 5 % NK, p = w / 5 / NK % kLallPl, t = w / 5 / NK / kLallPl;
    const size_t off = ((size_t)p * K + k) * kGallPl;
    const double a = A.aQp[t * n3p + off], av = -a * P.flxp[off + v];
    const PoleFace f = pole_face(P, t, p, k, v);
    atomicAdd(&A.a_flxp[off + v], -a * mx(mn(mn(mx(f.v0, f.lo), f.hi), f.bv[4]), f.bv[3]));
    if (av == 0.0) return;
    double *aq = A.a_qp + t * n3p + off, *ab = A.a_bb + (f.bv - P.bb);
    const Pick pick = limited(f.v0, f.lo, f.hi, f.bv[3], f.bv[4]);
    if (pick == kQmax || pick == kQmin) {
      atomicAdd(&ab[pick == kQmax ? 4 : 3], av);
    } else if (pick == kLow || pick == kHigh) {
      const int pt[4] = {0, v, (v == 1) ? 5 : v - 1, (v == 5) ? 1 : v + 1};
      const double qv[4] = {f.q[pt[0]], f.q[pt[1]], f.q[pt[2]], f.q[pt[3]]};
      atomicAdd(&aq[pt[arg4(qv, pick == kHigh)]], av);
    } else {
      atomicAdd(&aq[f.up], av);
      for (int d = 0; d < 3; ++d) {
        const size_t xi = d * n3p + off + v;
        atomicAdd(&ab[d], av * (P.xcp[xi] - P.GRD_xp[((size_t)d * kLallPl + p) * kGallPl + f.up]));
        atomicAdd(&A.a_xcp[xi], av * f.bv[d]);
      }
    }
    return;
  }
  const int e = (int)(u % P.ns), k = D.kmin - 1 + (int)(u / P.ns), code = P.seam[e];
  const int a = code % 3, o = code / 3 % D.gall, l = code / 3 / D.gall;
  const int i = o % G + 1, j = o / G + 1, nb = o + face_step(a, G);
  const bool inO = P.inner(i, j), inN = P.inner(a < 2 ? i + 1 : i, a > 0 ? j + 1 : j);
  if (!inO && !inN) return;  // no interior cell reads it
  const size_t off = ((size_t)l * K + k) * D.gall, gw = (size_t)D.lall * D.gall;
  const double *rho = P.rho + off;
  int p[4] = {o, 0, 0, 0};
  if (a == 0) {
    p[1] = max(o - G, 0), p[2] = o + 1, p[3] = o + G + 1;
  } else if (a == 1) {
    const bool sing = D.have_sgp[l] != 0 && i == D.gmin - 1 && j == D.gmin - 1;
    p[1] = sing ? o + G + 1 : o + 1, p[2] = sing ? o + G + 2 : o + G + 1, p[3] = o + G;
  } else {
    p[1] = o + G + 1, p[2] = o + G, p[3] = max(o - 1, 0);
  }
  const double fo = P.flx[a * n3 + off + o], fn = P.flx[(a + 3) * n3 + off + nb];
  const int up = upmask(fo, rho[o]) ? nb : o, b = P.bsrc[(size_t)l * D.gall + up];
  double disp[3], ax[3] = {0.0, 0.0, 0.0};
  for (int d = 0; d < 3; ++d) disp[d] = P.xc[(d * 3 + a) * n3 + off + o] - P.GRD_x[d * gw + (size_t)l * D.gall + up];
  for (int t = 0; t < P.nt; ++t) {
    const double *Q = P.Q + t * n3 + off, *aQ = A.aQ + t * n3 + off;
    const double t1 = inO ? -aQ[o] * fo : 0.0, t2 = inN ? -aQ[nb] * fn : 0.0, av = t1 + t2;
    if (av == 0.0) continue;
    const double qv[4] = {Q[p[0]] / rho[p[0]], Q[p[1]] / rho[p[1]], Q[p[2]] / rho[p[2]], Q[p[3]] / rho[p[3]]};
    const double qu = Q[up] / rho[up];
    // a halo point no list fills has no gradient, and Qout = q
    const double none[5] = {0.0, 0.0, 0.0, qu, qu}, *bv = b >= 0 ? P.bval(t, k, b) : none;
    double v0 = qu;
    for (int d = 0; d < 3; ++d) v0 = v0 + bv[d] * disp[d];
    const Pick pick = limited(v0, mn4(qv[0], qv[1], qv[2], qv[3]), mx4(qv[0], qv[1], qv[2], qv[3]), bv[3], bv[4]);
    double *aq = A.a_q + t * n3 + off;
    if (pick == kLow || pick == kHigh) {
      atomicAdd(&aq[p[arg4(qv, pick == kHigh)]], av);
    } else if (pick == kRemap) {
      atomicAdd(&aq[up], av);
      for (int d = 0; d < 3; ++d) {
        if (b >= 0) atomicAdd(A.abval(t, k, b) + d, av * disp[d]);
        ax[d] += av * bv[d];
      }
    } else if (b >= 0) {
      atomicAdd(A.abval(t, k, b) + (pick == kQmax ? 4 : 3), av);
    } else {
      atomicAdd(&aq[up], av);
    }
  }
  for (int d = 0; d < 3; ++d) {
    double &x = A.a_xc[(d * 3 + a) * n3 + off + o];
    x = A.first ? ax[d] : x + ax[d];
  }
}

// pole centre (t, p, k): Qout (mod_src_tracer.f90:307-367) and gradient, transposed
__device__ __forceinline__ void adj_pole_centre(const AdjArgs &A, int t, int p, int k) {
  const PlainArgs &P = A.P;
  const size_t off = ((size_t)p * P.D.kall + k) * kGallPl, n3p = P.n3p();
  const double *ab = A.abval(t, k, P.nb - 2 + p);
  double *a_q = A.a_qp + t * n3p + off;
  for (int x = 0; x < 3; ++x) {
    const double *cx = P.cgp + ((size_t)p * 3 + x) * 6;
    for (int v = 0; v < kGallPl; ++v) a_q[v] += cx[v] * ab[x];
  }
  const double aQn = ab[3], aQx = ab[4];
  if (aQn == 0.0 && aQx == 0.0) return;
  double qs[kGallPl], qmn[6], qmx[6], chm[6], ch[6];
  int pmn[6], pmx[6];
  for (int v = 0; v < kGallPl; ++v) qs[v] = P.Qp[t * n3p + off + v] / P.rhop[off + v];
  double qnmin = qs[0], qnmax = qs[0], Cin = 0.0, Cout = 0.0, CQmax = 0.0, CQmin = 0.0;
  int snmin = 0, snmax = 0;
  for (int v = 1; v <= 5; ++v) {
    const int pt[4] = {0, v, (v == 1) ? 5 : v - 1, (v == 5) ? 1 : v + 1};
    const double qv[4] = {qs[pt[0]], qs[pt[1]], qs[pt[2]], qs[pt[3]]};
    const bool in = upmask(P.flxp[off + v], P.rhop[off]);
    qmn[v] = in ? mn4(qv[0], qv[1], qv[2], qv[3]) : kBig;
    qmx[v] = in ? mx4(qv[0], qv[1], qv[2], qv[3]) : -kBig;
    pmn[v] = in ? pt[arg4(qv, false)] : -1;
    pmx[v] = in ? pt[arg4(qv, true)] : -1;
    if (qmn[v] < qnmin) qnmin = qmn[v], snmin = v;
    if (qmx[v] > qnmax) qnmax = qmx[v], snmax = v;
    ch[v] = P.flxp[off + v] / P.rhop[off];
    chm[v] = in ? ch[v] : 0.0;
    Cin = Cin + chm[v];
    Cout = Cout - chm[v] + ch[v];
    CQmin = CQmin + chm[v] * qmn[v];
    CQmax = CQmax + chm[v] * qmx[v];
  }
  if (0.5 - sgn(0.5, fabs(Cout) - kEps) != 0.0) {
    a_q[0] += aQn + aQx;
    return;
  }
  const double S = 1.0 - Cin - Cout, Dn = Cout;
  const double Nmn = qs[0] - CQmax - qnmax * S, Nmx = qs[0] - CQmin - qnmin * S;
  const double aNmn = aQn / Dn, aNmx = aQx / Dn, aD = -(aQn * Nmn + aQx * Nmx) / (Dn * Dn);
  const double a_qnmax = -aNmn * S, a_qnmin = -aNmx * S, aS = -aNmn * qnmax - aNmx * qnmin;
  const double aCQmax = -aNmn, aCQmin = -aNmx, aCin = -aS, aCout = -aS + aD;
  a_q[0] += aNmn + aNmx;
  a_q[snmax ? pmx[snmax] : 0] += a_qnmax;
  a_q[snmin ? pmn[snmin] : 0] += a_qnmin;
  for (int v = 1; v <= 5; ++v) {
    double achm = aCin - aCout;
    if (pmn[v] >= 0) {
      a_q[pmn[v]] += aCQmin * chm[v], a_q[pmx[v]] += aCQmax * chm[v];
      achm += aCQmin * qmn[v] + aCQmax * qmx[v];
    }
    atomicAdd(&A.a_chp[off + v], aCout + (pmn[v] >= 0 ? achm : 0.0));
  }
}

// The cells.  The upwind cell of a face holds every operand of its value, so the face, the remap, the
// cell's Qout and its gradient are transposed by that cell's thread: the adjoints of its gradient and
// Qout are registers, those of the tracer-independent inputs (fluxes, face centroids, Courant
// numbers) are summed over the tracers on chip, and a tracer's adjoint of q leaves as seven values a
// cell that the tile adds up in shared memory.  Only what a bound hands to one of its cells, which
// the data decide, goes to memory one by one (atomicAdd).
// Bound by latency at 12 warps an SM (168 registers and 75 KB a block): 1.9 ms for 8 tracers of glevel
// 6, kall 42; with the per-thread sums in registers two blocks fit and it took 2.3, or three that
// spilled, 3.0.
constexpr int kAdjCells = 128;  // threads, one per cell of a TX x (128 / TX) tile
constexpr int kAdjBlocks = 3;   // per SM

// cells bounding face f (0..5: faces 1-6, 6: face 5 of a singular corner) as neighbours of the cell, the
// owner first (mod_src_tracer.f90:152-214), and the neighbours' steps in i and j
__constant__ signed char kFacePts[7][4] = {{0, 6, 1, 2}, {0, 1, 2, 3}, {0, 2, 3, 4}, {4, 5, 0, 3},
                                           {5, 6, 0, 4}, {6, 1, 0, 5}, {5, 0, 1, 4}};
__constant__ signed char kStepI[7] = {0, 1, 1, 0, -1, -1, 0}, kStepJ[7] = {0, 0, 1, 1, 0, -1, -1};

template <int TX>
struct AdjCellSmem : CellSmem<TX, kAdjCells> {  // q[0]: q of the window, q[1]: adjoint of rhogq there
  double part[7][kAdjCells];  // adjoints of q of a cell and its neighbours
  // each thread's own, here for want of registers: fluxes of its faces and their adjoints, adjoints of
  // the chosen outflow faces' centroids and of the Courant numbers
  double flx[6][kAdjCells], aflx[6][kAdjCells], axc[9][kAdjCells], ach[6][kAdjCells];
};

template <int TX>
__global__ void __launch_bounds__(kAdjCells, kAdjBlocks) k_adj_cells(AdjArgs A, int ntx, int nty, int nlb, int lpb) {
  using Tile = CellTile<TX, kAdjCells>;
  using S = AdjCellSmem<TX>;
  extern __shared__ __align__(16) unsigned char raw[];
  S &s = *reinterpret_cast<S *>(raw);
  const PlainArgs &P = A.P;
  const Dims &D = P.D;
  const int G = D.gall_1d, tid = threadIdx.x, nmain = ntx * nty * D.lall * nlb;
  if ((int)blockIdx.x >= nmain) {
    const int u = ((int)blockIdx.x - nmain) * kAdjCells + tid, NK = D.kmax - D.kmin + 1;
    if (u < P.nt * kLallPl * NK) adj_pole_centre(A, u / NK / kLallPl, u / NK % kLallPl, D.kmin - 1 + u % NK);
    return;
  }
  const int lb = (int)blockIdx.x % nlb;
  Tile T;
  T.init(P, s, (int)blockIdx.x / nlb, ntx, nty);
  const int c = T.c;
  const size_t n3 = P.n3();
  const int k0 = D.kmin - 1 + lb * lpb, k1 = min(k0 + lpb, D.kmax);
  for (int k = k0; k < k1; ++k) {
    const size_t off = ((size_t)T.l * D.kall + k) * D.gall;
    double Qw[Tile::NSLOT][1], aw[Tile::NSLOT];
    auto load = [&](int t) {
      const double *Qs = P.Q + (size_t)t * n3 + off, *as = A.aQ + (size_t)t * n3 + off;
#pragma unroll
      for (int r = 0; r < Tile::NSLOT; ++r)
        if (T.wc[r] >= 0) Qw[r][0] = Qs[T.wc[r]], aw[r] = as[T.wc[r]];
    };
    load(0);
    CellFlow F;
    double fo[3];
    {
      Recip rw[Tile::NSLOT];
      double flx[6];
      T.level(P, s, off, rw, F, flx);
#pragma unroll
      for (int m = 0; m < 6; ++m) s.flx[m][tid] = flx[m], s.aflx[m][tid] = s.ach[m][tid] = 0.0;
#pragma unroll
      for (int m = 0; m < 9; ++m) s.axc[m][tid] = 0.0;
    }
    // the flux of the chosen outflow faces as their other cell has it, with this cell's own
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const bool f = (F.side >> a) & 1u;
      fo[a] = F.st[a] >= 0 ? (P.flx + (size_t)(f ? a : a + 3) * n3 + off)[f ? F.st[a] : c + face_step(a, G)] : 0.0;
      if (A.first && ((F.again >> a) & 1u))
        for (int d = 0; d < 3; ++d) (A.a_xc + (size_t)(d * 3 + a) * n3 + off)[c - face_step(a, G)] = 0.0;
    }
    for (int t = 0; t < P.nt; ++t) {
      double *a_q = A.a_q + (size_t)t * n3 + off;
#pragma unroll
      for (int r = 0; r < Tile::NSLOT; ++r)
        if (T.wc[r] >= 0) {
          const int e = tid + r * kAdjCells;
          const double rho = s.rho[e];
          quotients(Qw[r], Recip{rho, s.y[e], recip_ok(rho)});
          s.q[0][e] = Qw[r][0];
          s.q[1][e] = aw[r];
        }
      if (t + 1 < P.nt) load(t + 1);
      {  // the fluxes of the cell's faces, in Qh = Q - sum_m flx(m) fv(m)
        const double *fv = P.fv + (size_t)t * 3 * n3 + off, aH = T.act ? (A.aQ + (size_t)t * n3 + off)[c] : 0.0;
        const double f[6] = {fv[c], (fv + n3)[c], (fv + 2 * n3)[c], fv[c - 1], (fv + n3)[c - G - 1], (fv + 2 * n3)[c - G]};
#pragma unroll
        for (int m = 0; m < 6; ++m) s.aflx[m][tid] += -aH * f[m];
      }
      __syncthreads();
      double n[7], g[3];
      T.gradient(s, 0, n, g);
      CellLimits L;
      cell_limits(n, F, T.sing, L);
      double aself = 0.0, ag[3] = {0.0, 0.0, 0.0}, aQn = 0.0, aQx = 0.0;
      if (T.bs >= 0) {  // what seam and pole faces hand to this cell's values
        const double *o = A.abval(t, k, T.bs);
        ag[0] = o[0], ag[1] = o[1], ag[2] = o[2], aQn = o[3], aQx = o[4];
      }
      const double aH = s.q[1][T.ew];
      // the cell (as a neighbour of this one) that face f's lower or upper bound is a copy of
      auto bound = [&](int f, bool high) {
        const signed char *pt = kFacePts[(f == 4 && T.sing) ? 6 : f];
        int at = pt[0];
        double best = s.q[0][T.ew + kStepJ[at] * S::WW + kStepI[at]];
        for (int x = 1; x < 4; ++x) {
          const int q = pt[x];
          const double v = s.q[0][T.ew + kStepJ[q] * S::WW + kStepI[q]];
          if (high ? v > best : v < best) best = v, at = q;
        }
        return c + kStepJ[at] * G + kStepI[at];
      };
      // outflow face m (of faces a + 1 and a + 4): own flux fm, the other cell's fn and its adjoint aN
      auto face = [&](int a, int m, double lo, double hi, double fn, int slot, auto centroid) {
        const double fm = s.flx[m - 1][tid], aN = s.q[1][T.ew + (m > 3 ? Tile::wstep(a + 4) : Tile::wstep(a + 1))];
        const double av = -aH * fm + -aN * fn;
        if (av == 0.0) return;
        double v0 = n[0], disp[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) disp[d] = s.disp[a * 3 + d][slot], v0 = v0 + g[d] * disp[d];
        const Pick pick = limited(v0, lo, hi, L.Qmin, L.Qmax);
        if (pick == kRemap) {
          aself += av;
#pragma unroll
          for (int d = 0; d < 3; ++d) ag[d] += av * disp[d], centroid(d, av * g[d]);
        } else if (pick == kQmin) {
          aQn += av;
        } else if (pick == kQmax) {
          aQx += av;
        } else {
          atomicAdd(&a_q[bound(m - 1, pick == kHigh)], av);
        }
      };
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (F.st[a] < 0) continue;
        const bool f = (F.side >> a) & 1u;
        face(a, f ? a + 4 : a + 1, f ? L.lo[a + 4] : L.lo[a + 1], f ? L.hi[a + 4] : L.hi[a + 1], fo[a], F.sl[a],
             [&](int d, double x) { s.axc[a * 3 + d][tid] += x; });
      }
      if (F.again) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
          if ((F.again >> a) & 1u) {
            const int oc = c - face_step(a, G);
            face(a, a + 4, L.lo[a + 4], L.hi[a + 4], (P.flx + (size_t)a * n3 + off)[oc], T.ow - Tile::slot_back(a),
                 [&](int d, double x) { (A.a_xc + (size_t)(d * 3 + a) * n3 + off)[oc] += x; });
          }
      }
      // Qout (mod_src_tracer.f90:219-282): a cell whose bounds bind no face has nothing to hand on
      if (T.act && (aQn != 0.0 || aQx != 0.0)) {
        if (F.zsw) {
          aself += aQn + aQx;
        } else {
          const double Dn = F.den.b, O = F.omc;
          const double Nmn = n[0] - L.CQmax - L.qnmax * O, Nmx = n[0] - L.CQmin - L.qnmin * O;
          const double aNmn = aQn / Dn, aNmx = aQx / Dn, aD = -(aQn * Nmn + aQx * Nmx) / (Dn * Dn);
          const double aS = -aNmn * L.qnmax - aNmx * L.qnmin;
          const double aCQmax = -aNmn, aCQmin = -aNmx, aCin = -aS, aCout = -aS + aD;
          aself += aNmn + aNmx;
          int fmin = 0, fmax = 0;  // the face whose bound is qnmin / qnmax, 0: the cell itself
          double lowest = n[0], highest = n[0];
#pragma unroll
          for (int m = 1; m <= 6; ++m) {
            const bool f = (F.in >> m) & 1u;
            if (f && L.lo[m] < lowest) lowest = L.lo[m], fmin = m;
            if (f && L.hi[m] > highest) highest = L.hi[m], fmax = m;
            double achm = aCin;
            if (f) {
              atomicAdd(&a_q[bound(m - 1, false)], aCQmin * F.chm[m]);
              atomicAdd(&a_q[bound(m - 1, true)], aCQmax * F.chm[m]);
              achm += aCQmin * L.lo[m] + aCQmax * L.hi[m];
            }
            s.ach[m - 1][tid] += (s.flx[m - 1][tid] / s.rho[T.ew] > 0.0) ? aCout : achm;
          }
          if (fmax) atomicAdd(&a_q[bound(fmax - 1, true)], -aNmn * O);
          else aself += -aNmn * O;
          if (fmin) atomicAdd(&a_q[bound(fmin - 1, false)], -aNmx * O);
          else aself += -aNmx * O;
        }
      }
      // the gradient's stencil; the tile's cells are added up, one atomic per window cell
#pragma unroll
      for (int m = 0; m < 7; ++m) {
        double x = s.cg[m][tid] * ag[0];
        x += s.cg[7 + m][tid] * ag[1];
        x += s.cg[14 + m][tid] * ag[2];
        s.part[m][tid] = T.act ? (m == 0 ? aself + x : x) : 0.0;
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < Tile::NSLOT; ++r)
        if (T.wc[r] >= 0) {
          const int e = tid + r * kAdjCells, wx = e % S::WW - 1, wy = e / S::WW - 1;  // in the tile's frame
          double sum = 0.0;
#pragma unroll
          for (int m = 0; m < 7; ++m) {
            constexpr int DX[7] = {0, 1, 1, 0, -1, -1, 0}, DY[7] = {0, 0, 1, 1, 0, -1, -1};
            const int x = wx - DX[m], y = wy - DY[m];
            if (x >= 0 && x < TX && y >= 0 && y < S::TY) sum += s.part[m][y * TX + x];
          }
          if (sum != 0.0) atomicAdd(&a_q[T.wc[r]], sum);
        }
    }
    // ---- the level's sums over the tracers
    if (T.act) {
      const double rc = s.rho[T.ew], ah = A.last ? A.a_rh[off + c] : 0.0;
      double ar = ah;
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        const double a = s.ach[m][tid];
        double f = s.aflx[m][tid] - ah;
        if (a != 0.0) f += a / rc, ar += -a * (s.flx[m][tid] / rc) / rc;
        double &o = (A.a_flx + (size_t)m * n3 + off)[c];
        o = A.first ? f : o + f;
      }
      if (ar != 0.0) A.a_rho[off + c] += ar;
#pragma unroll
      for (int a = 0; a < 3; ++a)
        if (F.st[a] >= 0) {
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            double &o = (A.a_xc + (size_t)(d * 3 + a) * n3 + off)[F.st[a]];
            o = A.first ? s.axc[a * 3 + d][tid] : o + s.axc[a * 3 + d][tid];
          }
        }
    }
  }
}

// q = Q / rho: a_Q += a_q / rho, a_rho -= a_q q / rho, over the group's tracers (regions and poles in
// one launch, physical levels)
__global__ void __launch_bounds__(256) k_adj_div(AdjArgs A) {
  const PlainArgs &P = A.P;
  const Dims &D = P.D;
  const int NK = D.kmax - D.kmin + 1;
  const long long u = (long long)blockIdx.x * 256 + threadIdx.x, nreg = (long long)D.lall * NK * D.gall;
  const double *rho, *aq, *Q;
  double *aQ, *ar;
  size_t ts;
  if (u < nreg) {
    const size_t o = ((size_t)(u / D.gall / NK) * D.kall + D.kmin - 1 + u / D.gall % NK) * D.gall + u % D.gall;
    rho = P.rho + o, aq = A.a_q + o, Q = P.Q + o, aQ = A.aQ + o, ar = A.a_rho + o, ts = P.n3();
  } else {
    const int w = (int)(u - nreg);
    if (w >= kLallPl * NK * kGallPl) return;
    const size_t o = ((size_t)(w / kGallPl / NK) * D.kall + D.kmin - 1 + w / kGallPl % NK) * kGallPl + w % kGallPl;
    rho = P.rhop + o, aq = A.a_qp + o, Q = P.Qp + o, aQ = A.aQp + o, ar = A.a_rhop + o, ts = P.n3p();
  }
  const double r = *rho;
  double sum = 0.0;
  for (int t = 0; t < P.nt; ++t) {
    const double a = aq[t * ts];
    if (a == 0.0) continue;
    aQ[t * ts] += a / r;
    sum += -a * (Q[t * ts] / r) / r;
  }
  if (sum != 0.0) *ar += sum;
}

// pole centres: rho_h = rho - sum_m flx(m) and ch(m) = flx(m) / rho
__global__ void k_adj_rhoh_ch_pl(int kall, const double *rho_pl, const double *flx_pl, const double *a_rh_pl,
                                 const double *a_ch_pl, double *a_flx_pl, double *a_rho_pl) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= kLallPl * kall) return;
  const size_t off = (size_t)t * kGallPl;
  const double ah = a_rh_pl[off];
  a_rho_pl[off] += ah;
  for (int v = 2; v <= 6; ++v) a_flx_pl[off + v - 1] += -ah;
  const double r = rho_pl[off];
  for (int v = 2; v <= 6; ++v) {
    const double a = a_ch_pl[off + v - 1];
    if (a == 0.0) continue;
    a_flx_pl[off + v - 1] += a / r;
    a_rho_pl[off] += -a * (flx_pl[off + v - 1] / r) / r;
  }
}

// ---------------------------------------------------------------------------
// horizontal_flux.  Triangle values (:141-201): TI(ij) from (ij, ip1j, ip1jp1),
// TJ(ij) from (ij, ip1jp1, ijp1), TI(gmin-1,gmin-1) = TJ(gmin,gmin-1) on a
// singular region.  A face sums its two triangles: AI(ij) = TJ(ijm1) + TI(ij),
// AIJ(ij) = TI(ij) + TJ(ij), AJ(ij) = TJ(ij) + TI(im1j), and hands both of them the
// same adjoint, so each face is transposed once (k_adj_tri) and the fields gather from
// the faces of the six triangles around a point (k_adj_fields).  Both kernels stream a
// cell's levels with its weights and normals in registers, as the forward does, and ask
// for the next level's planes while a level is worked on: the latency of a level's loads
// bounds them.  One thread per triangle pair and level (each face transposed five times,
// twelve triangle values a cell) took 2.38 + 1.03 ms at glevel 7, kall 96; now 0.96 + 0.93.  At glevel 6,
// kall 42: 119 + 112 us a step, of 70 + 45 at the copy rate; k_adj_tri at 3 blocks per SM
// 136, without the prefetch 145, 5 blocks 206 (spills), 16 levels a thread 170;
// k_adj_fields without the prefetch 122.
constexpr int kAdjFluxThreads = 128, kAdjFluxLevels = 8;  // levels a thread

struct Fld {
  const double *f[4];  // rho, rhovx, rhovy, rhovz
};
struct Tv {
  double v[4];
};

__device__ __forceinline__ Tv tri(const Tv &f0, const Tv &f1, const Tv &f2, const double (&w)[3]) {
  Tv r;
#pragma unroll
  for (int x = 0; x < 4; ++x) r.v[x] = f0.v[x] * w[0] + f1.v[x] * w[1] + f2.v[x] * w[2];
  return r;
}

// A face's adjoint of its triangles' (rho, rhovx, rhovy, rhovz) sum: the wind parts take the place of
// a_xc, which nothing else reads any more, the density part goes to a_rs (3 fields); zero where a cell
// owns no face.  a_flx and a_xc hold what an interior cell on either side contributed; a face has them
// only there.  blocks: level blocks fastest, then cell blocks, then regions
__global__ void __launch_bounds__(kAdjFluxThreads, 4) k_adj_tri(Dims D, Geo<double> g, Fld F, const double *a_flx,
                                                               double *a_xc, double dt, double *a_rs, int lpb,
                                                               int nlb, int cellblk) {
  const int lb = (int)blockIdx.x % nlb, l = (int)blockIdx.x / nlb / cellblk;
  const int ci = (int)blockIdx.x / nlb % cellblk * kAdjFluxThreads + (int)threadIdx.x;
  if (ci >= D.gall) return;
  const int G = D.gall_1d, gmin = D.gmin, gmax = D.gmax;
  const int i = ci % G + 1, j = ci / G + 1;
  const unsigned c = ci;
  const size_t fs = (size_t)D.lall * D.kall * D.gall, gw = (size_t)D.gall * D.lall, lg = (size_t)l * D.gall;
  const bool sgp = D.have_sgp[l] != 0;
  const bool inI = i >= gmin && i <= gmax, inJ = j >= gmin && j <= gmax;
  const bool ext = i >= gmin - 1 && i <= gmax && j >= gmin - 1 && j <= gmax;
  const bool inO = inI && inJ;
  const bool inN[3] = {inner(D, i + 1, j), inner(D, i + 1, j + 1), inner(D, i, j + 1)};
  const bool face[3] = {ext && inJ && (inO || inN[0]), ext && (inO || inN[1]), ext && inI && (inO || inN[2])};
  const bool singI = sgp && i == gmin - 1 && j == gmin - 1, singJ = sgp && i == gmin && j == gmin - 1;
  double wI[3] = {}, wJ[3] = {}, wJm[3] = {}, wIm[3] = {}, wS[3] = {}, hn[3][3] = {}, ra[4] = {};
  if (ext) {
    auto weights = [&](int t, unsigned cell, double (&w)[3]) {
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
      for (int x = 0; x < 3; ++x) hn[a][x] = (g.GMTR_a + ((size_t)x * 3 + a) * gw + lg)[c];
    const double *rarea = g.GMTR_p + (size_t)(P_RAREA - 1) * gw + lg;
    ra[0] = rarea[c], ra[1] = rarea[c + 1], ra[2] = rarea[c + G + 1], ra[3] = rarea[c + G];
  }
  const int k0 = D.kmin - 1 + lb * lpb, k1 = min(k0 + lpb, D.kmax);  // the ghost levels have no part in the step
#pragma unroll 1
  for (int k = k0; k < k1; ++k) {
    const size_t off = ((size_t)l * D.kall + k) * D.gall;
    auto cell = [&](unsigned p) { return Tv{{(F.f[0] + off)[p], (F.f[1] + off)[p], (F.f[2] + off)[p], (F.f[3] + off)[p]}}; };
    if (k + 1 < k1) {
#pragma unroll
      for (int x = 0; x < 4; ++x) asm volatile("prefetch.global.L1 [%0];" ::"l"(F.f[x] + off + D.gall + c));
#pragma unroll
      for (int x = 0; x < 9; ++x) prefetch_l2(a_xc + (size_t)x * fs + off + D.gall + c);
#pragma unroll
      for (int x = 0; x < 6; ++x) prefetch_l2(a_flx + (size_t)x * fs + off + D.gall + c);
    }
    double afl[3] = {}, axc[3][3] = {};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const unsigned nb = c + (a == 0 ? 1 : (a == 1 ? G + 1 : G));
      if (!face[a]) continue;
      if (inO) afl[a] = (a_flx + (size_t)a * fs + off)[c] * ra[0] * dt;
      if (inN[a] && !(a == 2 && singJ)) afl[a] += -(a_flx + (size_t)(a + 3) * fs + off)[nb] * ra[a + 1] * dt;
#pragma unroll
      for (int x = 0; x < 3; ++x) axc[a][x] = (a_xc + ((size_t)x * 3 + a) * fs + off)[c];
    }
    Tv tI{}, tJ{}, tJm{}, tIm{};
    if (ext) {
      const Tv f00 = cell(c), f10 = cell(c + 1), f11 = cell(c + G + 1), f01 = cell(c + G);
      Tv f0m{}, fm0{};
      if (inJ) f0m = cell(c - G);
      if (inI) fm0 = cell(c - 1);
      tI = tri(f00, f10, f11, wI), tJ = tri(f00, f11, f01, wJ);
      tJm = tri(f0m, f10, f00, wJm), tIm = tri(fm0, f00, f01, wIm);
      if (singI) tI = tri(f10, cell(c + G + 2), f11, wS);
      if (singJ) tIm = tJ;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      double avs[3] = {}, ars = 0.0;
      if (face[a]) {
        const Tv &p = (a == 0) ? tJm : (a == 1 ? tI : tJ), &q = (a == 0) ? tI : (a == 1 ? tJ : tIm);
        const double rsum = p.v[0] + q.v[0], rr = 1.0 / mx(rsum, kEps);
        double arr = 0.0;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          const double ax = axc[a][x];
          avs[x] = 0.5 * afl[a] * hn[a][x];
          avs[x] += -ax * rr * dt * 0.5;
          arr += -ax * (p.v[x + 1] + q.v[x + 1]) * dt * 0.5;
        }
        ars = (rsum > kEps) ? -arr * rr * rr : 0.0;
      }
      (a_rs + (size_t)a * fs + off)[c] = ars;
#pragma unroll
      for (int x = 0; x < 3; ++x) (a_xc + ((size_t)x * 3 + a) * fs + off)[c] = avs[x];
    }
  }
}

// fields from the faces: point p is ij of TI/TJ(p) (W1), ip1j of TI(p-1) (W2),
// ip1jp1 of TI(p-G-1) (W3) and TJ(p-G-1) (W2), ijp1 of TJ(p-G) (W3); on a singular
// region TI(gmin-1,gmin-1) is TJ(gmin,gmin-1).  TI(c) has the faces AI(c), AIJ(c), AJ(c+1),
// TJ(c) the faces AIJ(c), AI(c+G), AJ(c)
__global__ void __launch_bounds__(kAdjFluxThreads) k_adj_fields(Dims D, const double *GT, const double *a_rs,
                                                               const double *a_xc, int lpb, int nlb, int cellblk,
                                                               double *a0, double *a1, double *a2, double *a3) {
  const int lb = (int)blockIdx.x % nlb, l = (int)blockIdx.x / nlb / cellblk;
  const int p = (int)blockIdx.x / nlb % cellblk * kAdjFluxThreads + (int)threadIdx.x;
  if (p >= D.gall) return;
  const int G = D.gall_1d, i = p % G + 1, j = p / G + 1;
  const size_t fs = (size_t)D.lall * D.kall * D.gall, gw = (size_t)D.gall * D.lall;
  const bool sgp = D.have_sgp[l] != 0;
  const int sg = (D.gmin - 2) * G + (D.gmin - 2);
  const bool i0 = i >= D.gmin - 1 && i <= D.gmax, j0 = j >= D.gmin - 1 && j <= D.gmax;  // p owns triangles
  const bool im = i >= D.gmin && i - 1 <= D.gmax, jm = j >= D.gmin && j - 1 <= D.gmax;  // ip-1, jp-1 do
  const bool ok[4] = {i0 && j0, im && j0, im && jm, i0 && jm};
  auto w = [&](bool on, int c, int t, int wi) {
    return on ? GT[((size_t)(wi - 1) * 2 + (t - 1)) * gw + (size_t)l * D.gall + c] : 0.0;
  };
  const double w0I = w(ok[0], p, TI, W1), w0J = w(ok[0], p, TJ, W1), w1I = w(ok[1], p - 1, TI, W2),
               w2I = w(ok[2], p - G - 1, TI, W3), w2J = w(ok[2], p - G - 1, TJ, W2), w3J = w(ok[3], p - G, TJ, W3);
  const int k0 = D.kmin - 1 + lb * lpb, k1 = min(k0 + lpb, D.kmax);
#pragma unroll 1
  for (int k = k0; k < k1; ++k) {
    const size_t off = ((size_t)l * D.kall + k) * D.gall;
    double sum[4];
    if (k + 1 < k1) {
#pragma unroll
      for (int x = 0; x < 9; ++x) prefetch_l2(a_xc + (size_t)x * fs + off + D.gall + p);
#pragma unroll
      for (int x = 0; x < 3; ++x) prefetch_l2(a_rs + (size_t)x * fs + off + D.gall + p);
    }
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      auto f = [&](int a, int c) { return ((x == 0 ? a_rs + (size_t)a * fs : a_xc + ((size_t)(x - 1) * 3 + a) * fs) + off)[c]; };
      auto sumI = [&](int c) { return f(0, c) + f(1, c) + f(2, c + 1); };
      auto aI = [&](int c) { return (sgp && c == sg) ? 0.0 : sumI(c); };
      auto aJ = [&](int c) {
        double v = f(1, c) + f(0, c + G) + f(2, c);
        if (sgp && c == sg + 1) v += sumI(sg);
        return v;
      };
      double s = 0.0;
      if (ok[0]) s += aI(p) * w0I + aJ(p) * w0J;
      if (ok[1]) s += aI(p - 1) * w1I;
      if (ok[2]) s += aI(p - G - 1) * w2I + aJ(p - G - 1) * w2J;
      if (ok[3]) s += aJ(p - G) * w3J;
      sum[x] = s;
    }
    a0[off + p] += sum[0], a1[off + p] += sum[1], a2[off + p] += sum[2], a3[off + p] += sum[3];
  }
}

// pole faces of horizontal_flux (:326-374), one thread per (pole, level)
__global__ void k_adj_flux_pl(int kall, Geo<double> g, Fld F, const double *a_flx_pl, const double *a_xc_pl,
                              double dt, double *a0, double *a1, double *a2, double *a3) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= kLallPl * kall) return;
  const int l = t / kall;
  const size_t off = (size_t)t * kGallPl, fsp = (size_t)kLallPl * kall * kGallPl;
  auto GT = [&](int v, int wi) { return g.GMTR_t_pl[((size_t)(wi - 1) * kLallPl + l) * kGallPl + (v - 1)]; };
  auto GA = [&](int v, int h) { return g.GMTR_a_pl[((size_t)(h - 1) * kLallPl + l) * kGallPl + (v - 1)]; };
  const double rarea = g.GMTR_p_pl[((size_t)(P_RAREA - 1) * kLallPl + l) * kGallPl + 0];
  double tt[7][4], at[7][4];
  for (int v = 2; v <= 6; ++v) {
    const int vp = (v == 6) ? 2 : v + 1;
    for (int x = 0; x < 4; ++x) {
      tt[v][x] = F.f[x][off] * GT(v, W1) + F.f[x][off + v - 1] * GT(v, W2) + F.f[x][off + vp - 1] * GT(v, W3);
      at[v][x] = 0.0;
    }
  }
  for (int v = 2; v <= 6; ++v) {
    const int vm = (v == 2) ? 6 : v - 1;
    const double rsum = tt[vm][0] + tt[v][0];
    const double rr = 1.0 / mx(rsum, kEps);
    const double aflux = a_flx_pl[off + v - 1] * rarea * dt;
    double avs[3], arr = 0.0;
    for (int x = 0; x < 3; ++x) avs[x] = 0.5 * aflux * GA(v, HNX + x);
    for (int x = 0; x < 3; ++x) {
      const double vsx = tt[vm][x + 1] + tt[v][x + 1];
      const double ax = a_xc_pl[(size_t)x * fsp + off + v - 1];
      avs[x] += -ax * rr * dt * 0.5;
      arr += -ax * vsx * dt * 0.5;
    }
    const double ars = (rsum > kEps) ? -arr * rr * rr : 0.0;
    at[vm][0] += ars, at[v][0] += ars;
    for (int x = 0; x < 3; ++x) at[vm][x + 1] += avs[x], at[v][x + 1] += avs[x];
  }
  double *out[4] = {a0, a1, a2, a3};
  for (int v = 2; v <= 6; ++v) {
    const int vp = (v == 6) ? 2 : v + 1;
    for (int x = 0; x < 4; ++x) {
      out[x][off] += at[v][x] * GT(v, W1);
      out[x][off + v - 1] += at[v][x] * GT(v, W2);
      out[x][off + vp - 1] += at[v][x] * GT(v, W3);
    }
  }
}

template <int TX>
cudaError_t launch_adj_cells(const AdjArgs &A, cudaStream_t st) {
  const Dims &D = A.P.D;
  using S = AdjCellSmem<TX>;
  const int n = D.gmax - D.gmin + 1, ntx = (n + TX - 1) / TX, nty = (n + S::TY - 1) / S::TY;
  const int tiles = ntx * nty * D.lall, NK = D.kmax - D.kmin + 1;
  int lpb = 8;  // levels a block, as in the forward's cell kernel
  while (lpb > 1 && (long long)tiles * ((NK + lpb - 1) / lpb) < 2 * kAdjBlocks * 148) lpb /= 2;
  const int nlb = (NK + lpb - 1) / lpb, npole = (A.P.nt * kLallPl * NK + kAdjCells - 1) / kAdjCells;
  cudaError_t e = cudaFuncSetAttribute(k_adj_cells<TX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(S));
  if (e != cudaSuccess) return e;
  k_adj_cells<TX><<<(unsigned)(tiles * nlb + npole), kAdjCells, sizeof(S), st>>>(A, ntx, nty, nlb, lpb);
  return cudaGetLastError();
}

void fill_adj(const StepCtx &S, double *a, double *a_pl, int vmax, cudaStream_t st) {
  const Dims &D = S.D;
  const long long total = (long long)S.plan.n * D.kall * vmax;
  if (total == 0) return;
  k_fill_adj<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(S.plan.n, S.plan.dst, S.plan.src, D.gall * D.lall,
                                                              D.gall, D.lall, D.kall, vmax, a, a_pl);
}

}  // namespace

int step_adjoint(StepCtx &S, const AdjScratch &A, int ntr, double dt, const double *rhog, const double *rhog_pl,
                 const double *rhogq, const double *rhogq_pl, const double *vx, const double *vx_pl,
                 const double *vy, const double *vy_pl, const double *vz, const double *vz_pl, const double *w,
                 const double *w_pl, double *a_rhog, double *a_rhog_pl, double *a_rhogq, double *a_rhogq_pl,
                 double *a_vx, double *a_vx_pl, double *a_vy, double *a_vy_pl, double *a_vz, double *a_vz_pl,
                 cudaStream_t st, long long &launches) {
  const Dims &D = S.D;
  if (D.kall < 4 || D.kmax <= D.kmin) return set_error("adjoint: bad vertical grid"), ICA_ERR_ARG;
  const size_t n3 = (size_t)D.gall * D.kall * D.lall, n3p = (size_t)kGallPl * D.kall * kLallPl;
  const size_t B = sizeof(double);
  const int T = 128, n = D.gmax - D.gmin + 1, NK = D.kmax - D.kmin + 1;
  const unsigned nbl = (unsigned)((kLallPl * D.kall + 127) / 128);
  // ---- the step-level forward values, the final halo fill, the density part of the vertical sub-step
  FluxIn<double> fin{rhog, rhog_pl, vx, vx_pl, vy, vy_pl, vz, vz_pl};
  FluxOut<double> fout{S.flx, S.flx_pl, S.xc, S.xc_pl};
  launch_horizontal_flux<double>(D, fin, fout, S.geo, dt, st);
  cudaMemsetAsync(A.a_flx_pl, 0, n3p * B, st);
  cudaMemsetAsync(A.a_xc_pl, 0, 3 * n3p * B, st);
  cudaMemsetAsync(A.a_ch_pl, 0, n3p * B, st);
  fill_adj(S, a_rhog, a_rhog_pl, 1, st);
  fill_adj(S, a_rhogq, a_rhogq_pl, ntr, st);
  const int npt = D.lall * D.gall + kLallPl * kGallPl;
  k_adj_vrho<<<(npt + 127) / 128, 128, 0, st>>>(D, a_rhog, a_rhog_pl, A.a_rh, A.a_rh_pl);
  launches += 4;
  // ---- the tracers, a group at a time: recompute the faces, then transpose the two sub-steps
  for (int t0 = 0; t0 < ntr; t0 += kPlainGroup) {
    AdjArgs a{};
    // the forward's launches only read rhogq here
    a.P = plain_group(S, t0, ntr, dt, rhog, rhog_pl, const_cast<double *>(rhogq), const_cast<double *>(rhogq_pl), w, w_pl);
    const int nt = a.P.nt;
    a.aQ = a_rhogq + t0 * n3, a.aQp = a_rhogq_pl + t0 * n3p;
    a.Qh = A.a_q, a.Qhp = A.Qh_pl, a.a_q = A.a_q, a.a_qp = A.a_q_pl, a.a_bb = A.a_bb;
    a.rh = A.rh, a.rhp = A.rh_pl, a.a_rh = A.a_rh, a.a_rhp = A.a_rh_pl;
    a.a_flx = A.a_flx, a.a_flxp = A.a_flx_pl, a.a_xc = A.a_xc, a.a_xcp = A.a_xc_pl, a.a_chp = A.a_ch_pl;
    a.a_rho = a_rhog, a.a_rhop = a_rhog_pl;
    a.first = t0 == 0, a.last = t0 + nt >= ntr;
    const int rc = plain_faces(a.P, st, launches);
    if (rc) return rc;
    const int cellblk = (D.gall + T - 1) / T, nqh = cellblk * D.kall * D.lall;
    k_adj_qh<<<(unsigned)(nqh + (nt * kLallPl * D.kall + T - 1) / T), T, 0, st>>>(a, cellblk, nqh);
    // vertical sub-step: aQ becomes the adjoint of rhogq after the horizontal sub-step
    const int colblk = (n * n + kAdjThreads - 1) / kAdjThreads, ncol = colblk * D.lall * nt;
    k_adj_vert<<<(unsigned)(ncol + (nt * kLallPl + kAdjThreads - 1) / kAdjThreads), kAdjThreads, sizeof(AdjRing), st>>>(
        a, colblk, ncol);
    cudaMemsetAsync(A.a_q, 0, nt * n3 * B, st);
    cudaMemsetAsync(A.a_q_pl, 0, nt * n3p * B, st);
    cudaMemsetAsync(A.a_bb, 0, (size_t)nt * D.kall * S.nb * 5 * B, st);
    const long long nsm = (long long)S.ns * NK + (long long)kLallPl * NK * 5 * nt;
    k_adj_seam<<<(unsigned)((nsm + 127) / 128), 128, 0, st>>>(a);
    const cudaError_t e = n >= 32 ? launch_adj_cells<32>(a, st) : launch_adj_cells<16>(a, st);
    if (e != cudaSuccess) return set_error(std::string("adjoint: ") + cudaGetErrorString(e)), ICA_ERR_CUDA;
    const long long nd = (long long)NK * (D.lall * D.gall + kLallPl * kGallPl);
    k_adj_div<<<(unsigned)((nd + 255) / 256), 256, 0, st>>>(a);
    launches += 5;
  }
  // ---- the poles' density update and Courant numbers, then horizontal_flux
  k_adj_rhoh_ch_pl<<<nbl, 128, 0, st>>>(D.kall, rhog_pl, S.flx_pl, A.a_rh_pl, A.a_ch_pl, A.a_flx_pl, a_rhog_pl);
  const Fld F{{rhog, vx, vy, vz}};
  const Fld Fp{{rhog_pl, vx_pl, vy_pl, vz_pl}};
  {
    const int cb = (D.gall + kAdjFluxThreads - 1) / kAdjFluxThreads;
    int lpb = kAdjFluxLevels;  // fewer where the blocks would not fill the SMs
    while (lpb > 1 && (long long)cb * D.lall * ((NK + lpb - 1) / lpb) < 4 * 148) lpb /= 2;
    const int nlb = (NK + lpb - 1) / lpb;
    const unsigned nb = (unsigned)(cb * D.lall * nlb);
    k_adj_tri<<<nb, kAdjFluxThreads, 0, st>>>(D, S.geo, F, A.a_flx, A.a_xc, dt, A.a_rs, lpb, nlb, cb);
    k_adj_fields<<<nb, kAdjFluxThreads, 0, st>>>(D, S.geo.GMTR_t, A.a_rs, A.a_xc, lpb, nlb, cb, a_rhog, a_vx, a_vy, a_vz);
  }
  k_adj_flux_pl<<<nbl, 128, 0, st>>>(D.kall, S.geo, Fp, A.a_flx_pl, A.a_xc_pl, dt, a_rhog_pl, a_vx_pl, a_vy_pl,
                                     a_vz_pl);
  launches += 4;
  return ICA_OK;
}

}  // namespace icoadv
