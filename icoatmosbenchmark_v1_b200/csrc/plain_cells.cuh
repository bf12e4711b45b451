// What the plain step's kernels and their adjoint share: the arguments of a group of tracers, and the
// cell side of the horizontal sub-step (a tile of cells, one thread each, q of the tile and its ring
// in shared memory).
#pragma once

#include <cuda_runtime.h>

#include <cfloat>

#include "quotients.cuh"
#include "step.cuh"

namespace icoadv {

__device__ __forceinline__ double sgn(double a, double b) { return copysign(fabs(a), b); }

struct PlainArgs {
  Dims D;
  int nt, nb, ns;                    // tracers of the group; boundary entries, seam faces
  double dt;
  double *Q, *Qp;                    // the group's rhogq
  const double *rho, *rhop, *w, *wp, *flx, *flxp, *xc, *xcp;
  const double *GRD_x, *GRD_xp, *cg, *cgp, *rdgz, *afact, *bfact;
  const int *bsrc, *seam, *ring;     // boundary entry of a point, seam face codes, pole ring's entries
  double *fv;                        // (nt, 3, lall, kall, gall): limited values of faces AI, AIJ, AJ of their owner
  double *bb;                        // (nt, kall, nb, 5): gradient x/y/z, Qout min / max
  __device__ size_t n3() const { return (size_t)D.lall * D.kall * D.gall; }
  __device__ size_t n3p() const { return (size_t)kLallPl * D.kall * kGallPl; }
  __device__ double *bval(int t, int k, int b) const { return bb + (((size_t)t * D.kall + k) * nb + b) * 5; }
  __device__ bool inner(int i, int j) const { return i >= D.gmin && i <= D.gmax && j >= D.gmin && j <= D.gmax; }
};

__device__ __forceinline__ double mn(double a, double b) { return (b < a) ? b : a; }
__device__ __forceinline__ double mx(double a, double b) { return (b > a) ? b : a; }
__device__ __forceinline__ double mn4(double a, double b, double c, double d) { return mn(mn(mn(a, b), c), d); }
__device__ __forceinline__ double mx4(double a, double b, double c, double d) { return mx(mx(mx(a, b), c), d); }
// cmask of the Courant number f / r: true where it is 1 (the face's neighbour is its upwind cell),
// which is where the rounded quotient is below EPS.  EPS is a power of two, so for an ordinary
// density that is f < EPS r, without the division.
__device__ __forceinline__ bool upmask(double f, double r) {
  if (r >= 0x1p-900) return f < DBL_EPSILON * r;
  return 0.5 - sgn(0.5, f / r - DBL_EPSILON) != 0.0;
}

// cell index from the owner of face a (AI, AIJ, AJ) to its other cell
__device__ __forceinline__ int face_step(int a, int G) { return a == 0 ? 1 : (a == 1 ? G + 1 : G); }

// The tracer-independent part of a cell and level: Courant numbers, upwind sides, outflow sums.
struct CellFlow {
  double chm[7], omc;   // inflow Courant numbers of faces 1-6; 1 - Cin - Cout
  Recip den;            // Cout + zerosw
  bool zsw, odd;        // odd: an inflow Courant number at a face whose mask says outflow (rounding-level fluxes)
  unsigned in;          // bit m: face m is an inflow face
  // Of two opposite faces a + 1 and a + 4 a cell usually has one outflow face (between two interior
  // cells): side tells which, sl / st are its owner's slot and cell (st < 0: none).  Bits of again:
  // both flow out, and a + 4 is the second one.
  unsigned side, again;
  int sl[3], st[3];
};

// Bounds and Qout of a cell for one tracer.
struct CellLimits {
  double lo[7], hi[7], qnmin, qnmax, CQmin, CQmax, Qmin, Qmax;
};

// n: q of the cell and its neighbours (i+1,j), (i+1,j+1), (i,j+1), (i-1,j), (i-1,j-1), (i,j-1)
__device__ __forceinline__ void cell_limits(const double (&n)[7], const CellFlow &F, bool sing, CellLimits &L) {
  const double c0 = n[0], n1 = n[1], n2 = n[2], n3 = n[3], n4 = n[4], n5 = n[5], n6 = n[6];
  // 4-point bounds of the six faces (mod_src_tracer.f90:152-214): the cell and three
  // consecutive neighbours, of which each pair is compared once
  const double l12 = mn(n1, n2), l34 = mn(n3, n4), l56 = mn(n5, n6);
  const double h12 = mx(n1, n2), h34 = mx(n3, n4), h56 = mx(n5, n6);
  L.lo[1] = mn(c0, mn(n6, l12)), L.hi[1] = mx(c0, mx(n6, h12));
  L.lo[2] = mn(c0, mn(l12, n3)), L.hi[2] = mx(c0, mx(h12, n3));
  L.lo[3] = mn(c0, mn(n2, l34)), L.hi[3] = mx(c0, mx(n2, h34));
  L.lo[4] = mn(c0, mn(l34, n5)), L.hi[4] = mx(c0, mx(h34, n5));
  L.lo[5] = mn(c0, mn(n4, l56)), L.hi[5] = mx(c0, mx(n4, h56));
  L.lo[6] = mn(c0, mn(l56, n1)), L.hi[6] = mx(c0, mx(h56, n1));
  // Qout (:219-282, d = 0).  An outflow face's +-BIG bound never binds, and its term of CQ is
  // zero with its Courant number, except at an odd face
  double qnmin = c0, qnmax = c0, CQmin = F.chm[1] * L.lo[1], CQmax = F.chm[1] * L.hi[1];
#pragma unroll
  for (int m = 1; m <= 6; ++m) {
    const bool f = (F.in >> m) & 1u;
    qnmin = (f && L.lo[m] < qnmin) ? L.lo[m] : qnmin;
    qnmax = (f && L.hi[m] > qnmax) ? L.hi[m] : qnmax;
    if (m > 1) CQmin = CQmin + F.chm[m] * L.lo[m], CQmax = CQmax + F.chm[m] * L.hi[m];
  }
  if (F.odd || sing) {
    if (sing) L.lo[5] = mn4(n5, c0, n1, n4), L.hi[5] = mx4(n5, c0, n1, n4);  // the singular point's shifted stencil
    qnmin = qnmax = c0;
#pragma unroll
    for (int m = 1; m <= 6; ++m) {
      const bool f = (F.in >> m) & 1u;
      qnmin = (f && L.lo[m] < qnmin) ? L.lo[m] : qnmin;
      qnmax = (f && L.hi[m] > qnmax) ? L.hi[m] : qnmax;
      const double tmin = F.chm[m] * (f ? L.lo[m] : DBL_MAX), tmax = F.chm[m] * (f ? L.hi[m] : -DBL_MAX);
      CQmin = (m == 1) ? tmin : CQmin + tmin;
      CQmax = (m == 1) ? tmax : CQmax + tmax;
    }
  }
  double Qo[2] = {c0 - CQmax - qnmax * F.omc, c0 - CQmin - qnmin * F.omc};
  quotients(Qo, F.den);
  L.Qmin = F.zsw ? c0 : Qo[0], L.Qmax = F.zsw ? c0 : Qo[1];
  L.qnmin = qnmin, L.qnmax = qnmax, L.CQmin = CQmin, L.CQmax = CQmax;
}

// store x to p where on, without a branch
__device__ __forceinline__ void store_if(bool on, double *p, double x) {
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q st.global.f64 [%0], %1;\n}\n" ::"l"(p), "d"(x), "r"((int)on)
               : "memory");
}
__device__ __forceinline__ void prefetch_l2(const double *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

template <int TX, int NTH>
struct CellSmem {
  static constexpr int TY = NTH / TX, WW = TX + 2, NW = WW * (TY + 2);  // window: the tile and one ring
  static constexpr int OW = TX + 1, NO = OW * (TY + 1);                 // owners of the tile's faces
  double cg[21][NTH];
  // xc of the face [face * 3 + x][owner]; its upwind cell's thread turns it into xc - x(upwind cell)
  // and is the one that reads it
  double disp[9][NO];
  double rho[NW], y[NW];  // rhog and its reciprocal
  double q[2][NW];
};

// One thread's cell of a TX x (NTH / TX) tile.
template <int TX, int NTH>
struct CellTile {
  using Smem = CellSmem<TX, NTH>;
  static constexpr int NSLOT = (Smem::NW + NTH - 1) / NTH;  // window cells a thread fills
  static __device__ constexpr int slot_back(int a) { return a == 0 ? 1 : (a == 1 ? Smem::OW + 1 : Smem::OW); }
  static __device__ constexpr int wstep(int m) {  // window slots from a cell to its neighbour m
    return m == 0 ? 0 : m == 1 ? 1 : m == 2 ? Smem::WW + 1 : m == 3 ? Smem::WW : m == 4 ? -1 : m == 5 ? -Smem::WW - 1 : -Smem::WW;
  }
  // window slot r of this thread holds a cell (the first one always in a region of whole tiles)
  __device__ __forceinline__ bool has(int r) const { return (TX == 32 && r == 0) || wc[r] >= 0; }
  int l, c, ew, ow, bs, oslot, ocell, wc[NSLOT];
  bool act, sing;
  unsigned both;  // bit m: the cell across face m is interior too (not a seam face)
  double X[3];

  __device__ __forceinline__ void init(const PlainArgs &P, Smem &s, int tile, int ntx, int nty) {
    const Dims &D = P.D;
    const int G = D.gall_1d, tid = threadIdx.x, tr = tile % (ntx * nty);
    l = tile / (ntx * nty);
    const int i0 = D.gmin + (tr % ntx) * TX, j0 = D.gmin + (tr / ntx) * Smem::TY;  // first cell, 1-based
    const int i = i0 + tid % TX, j = j0 + tid / TX;
    // regions 32 or more cells wide are whole tiles; in a smaller one a thread without a cell works on
    // the region's last cell and stores nothing
    act = TX == 32 || (i <= D.gmax && j <= D.gmax);
    const int ci = TX == 32 ? i : min(i, D.gmax), cj = TX == 32 ? j : min(j, D.gmax);
    c = (cj - 1) * G + (ci - 1);
    sing = D.have_sgp[l] != 0 && ci == D.gmin && cj == D.gmin;
    const size_t gw = (size_t)D.lall * D.gall, lg = (size_t)l * D.gall;
    bs = act ? P.bsrc[lg + c] : -1;
#pragma unroll
    for (int n = 0; n < 21; ++n) s.cg[n][tid] = P.cg[((size_t)l * 21 + n) * D.gall + c];
    // this thread's window slots and their cells (-1: none)
#pragma unroll
    for (int r = 0; r < NSLOT; ++r) {
      const int e = tid + r * NTH, wi = i0 - 1 + e % Smem::WW, wj = j0 - 1 + e / Smem::WW;  // >= 1
      wc[r] = (e < Smem::NW && wi <= G && wj <= G) ? (wj - 1) * G + (wi - 1) : -1;
    }
    // owner slots of the faces: this cell's, and for the first threads one of the row and column
    // before the tile
    const int cx = ci - i0, cy = cj - j0;
    ew = (cy + 1) * Smem::WW + cx + 1, ow = (cy + 1) * Smem::OW + cx + 1;
    oslot = -1, ocell = 0;
    if (tid < TX + Smem::TY + 1) {
      const int ox = tid <= TX ? tid - 1 : -1, oy = tid <= TX ? -1 : tid - TX - 1;
      if (i0 + ox <= D.gmax && j0 + oy <= D.gmax)
        oslot = (oy + 1) * Smem::OW + ox + 1, ocell = (j0 + oy - 1) * G + (i0 + ox - 1);
    }
    constexpr int DX[7] = {0, 1, 1, 0, -1, -1, 0}, DY[7] = {0, 0, 1, 1, 0, -1, -1};
    both = 0;
#pragma unroll
    for (int m = 1; m <= 6; ++m) both |= act && P.inner(ci + DX[m], cj + DY[m]) ? 1u << m : 0u;
#pragma unroll
    for (int d = 0; d < 3; ++d) X[d] = P.GRD_x[d * gw + lg + c];
  }

  // A level's set-up (slab at off): the window's density, its reciprocals (also rw, this thread's
  // slots), the cell's flow and the displacements of its outflow faces.
  __device__ __forceinline__ void level(const PlainArgs &P, Smem &s, size_t off, Recip (&rw)[NSLOT], CellFlow &F,
                                        double (&flx)[6]) {
    const int G = P.D.gall_1d, tid = threadIdx.x;
    const size_t n3 = P.n3();
    double ch[6], fo[3], rv[NSLOT];
    const double *fx = P.flx + off;
#pragma unroll
    for (int m = 0; m < 6; ++m) ch[m] = flx[m] = (fx + m * n3)[c];
    fo[0] = fx[c - 1], fo[1] = (fx + n3)[c - G - 1], fo[2] = (fx + 2 * n3)[c - G];  // owners of faces 4-6
#pragma unroll
    for (int r = 0; r < NSLOT; ++r) rv[r] = has(r) ? P.rho[off + wc[r]] : 1.0;
    __syncthreads();  // the previous level's shared data is read
    const double *xc = P.xc + off;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        if (act) s.disp[a * 3 + d][ow] = (xc + (d * 3 + a) * n3)[c];
        if (oslot >= 0) s.disp[a * 3 + d][oslot] = (xc + (d * 3 + a) * n3)[ocell];
      }
#pragma unroll
    for (int r = 0; r < NSLOT; ++r) {
      rw[r] = recip(rv[r]);
      if (has(r)) s.rho[tid + r * NTH] = rv[r], s.y[tid + r * NTH] = rw[r].y;
    }
    __syncthreads();
    unsigned out = 0;
    F.in = 0, F.odd = false;
    const double rc = s.rho[ew];
#pragma unroll
    for (int m = 1; m <= 6; ++m) {
      // the owner's mask: 1 takes the owner's neighbour as the upwind cell
      const bool cm = (m <= 3) ? upmask(ch[m - 1], rc) : upmask(fo[m - 4], s.rho[ew + wstep(m)]);
      if (cm == (m <= 3)) F.in |= 1u << m;
      else if ((both >> m) & 1u) out |= 1u << m;
    }
    quotients(ch, Recip{rc, s.y[ew], recip_ok(rc)});
    F.chm[0] = 0.0;
#pragma unroll
    for (int m = 1; m <= 6; ++m) {
      F.chm[m] = mn(ch[m - 1], 0.0);
      F.odd = F.odd || (!((F.in >> m) & 1u) && F.chm[m] != 0.0);
    }
    const double *hm = F.chm;
    const double Cin = hm[1] + hm[2] + hm[3] + hm[4] + hm[5] + hm[6];
    const double Cout = ch[0] - hm[1] + ch[1] - hm[2] + ch[2] - hm[3] + ch[3] - hm[4] + ch[4] - hm[5] + ch[5] - hm[6];
    const double dv = 0.0, z = 0.5 - sgn(0.5, fabs(Cout) - DBL_EPSILON);
    F.zsw = z != 0.0;
    F.den = recip(Cout + z);
    F.omc = 1.0 - Cin - Cout + dv;
    F.side = F.again = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int so = ow - slot_back(a);
      const bool o1 = (out >> (a + 1)) & 1u, o2 = (out >> (a + 4)) & 1u;
      if (!o1 && o2) F.side |= 1u << a;
      if (o1 && o2) F.again |= 1u << a;
      F.sl[a] = (!o1 && o2) ? so : ow;
      F.st[a] = o1 ? c : (o2 ? c - face_step(a, G) : -1);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        if (o1 || o2) s.disp[a * 3 + d][F.sl[a]] -= X[d];
        if (o1 && o2) s.disp[a * 3 + d][so] -= X[d];
      }
    }
  }

  // asks L2 for the next level's set-up inputs and its first tracer's q
  __device__ __forceinline__ void prefetch(const PlainArgs &P, size_t off) const {
    const size_t n3 = P.n3();
#pragma unroll
    for (int m = 0; m < 6; ++m) prefetch_l2(P.flx + m * n3 + off + c);
#pragma unroll
    for (int m = 0; m < 9; ++m) prefetch_l2(P.xc + m * n3 + off + c);
    prefetch_l2(P.rho + off + c);
    prefetch_l2(P.Q + off + c);
  }

  // q of the cell and its neighbours from buffer b of the window, and the cell's gradient
  __device__ __forceinline__ void gradient(const Smem &s, int b, double (&n)[7], double (&g)[3]) const {
#pragma unroll
    for (int m = 0; m < 7; ++m) n[m] = s.q[b][ew + wstep(m)];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      g[d] = s.cg[d * 7][threadIdx.x] * n[0];
#pragma unroll
      for (int m = 1; m < 7; ++m) g[d] = g[d] + s.cg[d * 7 + m][threadIdx.x] * n[m];
    }
  }
};

// The group of tracers from t0 on, and its limited face values (fv) and boundary values (bb).
PlainArgs plain_group(const StepCtx &S, int t0, int ntr, double dt, const double *rhog, const double *rhog_pl,
                      double *rhogq, double *rhogq_pl, const double *w, const double *w_pl);
int plain_faces(const PlainArgs &P, cudaStream_t st, long long &launches);

}  // namespace icoadv
