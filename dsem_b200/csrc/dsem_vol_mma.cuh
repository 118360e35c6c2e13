// dsem_vol_mma.cuh -- volume kernel for elements with diagonal metrics (the
// axis-aligned hex elements of DSEM's boxes), p = 3..8, with the line
// contractions on the FP64 matrix instruction (mma.sync m8n8k4 f64, DMMA).
//
// Same mathematics and the same floating-point evaluation order as k_vol
// (Int_fluxes, Vis_Fluxes, Gauss_Deriv, update_interior:
// fluxesH_newa.f90:221-355, Vis_Fluxes_new.f90:16-382, SolnDerivsc.f90:14-83,
// updatea.f90:100-113): a DMMA runs the scalar contraction's FMA chain, in
// increasing k from its accumulator, so the two kernels agree bit for bit.
//
// What bounds it: the FP64 pipe, which DMMA and DFMA share at 64 FMAs per clock
// and SM.  A thread-per-point kernel reads every line value from shared memory once
// per Lobatto point (24.7k shared-memory wavefronts per element at p = 8 against
// 15.3k cycles of FP64 work) and passes Lobatto states and fluxes between phases
// through it.  Here a warp takes 8 lines of a direction at once: rows of the
// fragments are lines, columns their interior Lobatto points, so that every value
// is loaded once per line, and
//
//  pass 1  per (direction, tile): the Lobatto lines of rho, rho u, rho v, rho w
//          are interpolated, differentiated and scaled by gmetg(D,D) in registers;
//          the Gauss gradients go to shared memory (12 fields);
//  pass 2  per direction (z, y, x) and tile: the state and the 11 gradient fields
//          the direction needs are interpolated; each lane then holds its line at
//          s = 1+q and 5+q, evaluates both fluxes there, and its fluxes are already
//          the A fragment of the divergence contraction (the columns of the
//          interpolation are permuted so that they are).  No Lobatto array and no
//          flux is written to memory.  Face points are separate tasks, one line per
//          lane; the energy gradient is needed on its own grid only and is formed
//          one direction ahead.
// The divergence sums of the directions are added at L2 in the order z, y, x.
//
// Measured (22^3 elements of p = 8, the volume launch): 1.757 -> 1.127 ms; p = 7,
// 20^3: 1.286 -> 0.492; p = 6, 24^3: 1.088 -> 0.745; p = 5, 24^3: 0.568 -> 0.526;
// p = 4, 32^3: 0.717 -> 0.638; p = 3, 32^3: 0.372 -> 0.310.
#pragma once
#include "dsem_shapes.h"
#include "dsem_stage.cuh"

namespace dsem {

// D (8 x 8) += A (8 x 4) B (4 x 8).  Lane r*4+q holds A[r][q], B[q][r] and the
// accumulators D[r][2q], D[r][2q+1].
__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

// smallest plane stride >= G^2 congruent to 4 or 12 mod 16 doubles: the four
// k-lanes of a fragment along z, and the four rows of one across z, then fall
// into different banks
__host__ __device__ constexpr int mma_plane(int G) {
  int s = G * G;
  while (s % 16 != 4 && s % 16 != 12) ++s;
  return s;
}

template <int G, int V> struct MmaCfg {
  static constexpr int L = G + 1, G2 = G * G, NG = G * G * G, NL = L * G * G;
  static constexpr int PS = mma_plane(G), FS = G * PS;  // padded plane and field strides
  static constexpr int NS = G - 1;                      // interior Lobatto points s = 1..NS
  static constexpr int NI = NS > 4 ? 2 : 1;             // interior points per lane: s = 1+q, 5+q
  static constexpr int KF = G / 4, KR = G % 4;          // full k-steps and remaining k of a Gauss contraction
  static constexpr int KM = KR == 3 ? KF + 1 : KF;      // k-steps on the matrix unit (a remainder of 3 padded)
  static constexpr int KS = KR == 3 ? 0 : KR;           // k on scalar FMAs
  static constexpr int NTILE = (G2 + 7) / 8;            // tiles of 8 lines per direction
  static constexpr int NLW = (G2 + 31) / 32;            // warps of one line per lane
  static constexpr int NW = mma_warps(G, V), NT = 32 * NW;
  static constexpr int MINB = mma_minb(G, V);
  // shared fields: state 5, gradients of fields 0..3 12, energy gradient 2 buffers (general metrics: 5, 15)
  static constexpr int NF = V == MMA_GEN || V == MMA_GEN_WIDE ? 20 : 19;
  static constexpr size_t SMEM = sizeof(double) * (size_t)(NF * FS) + 16;
};

// Operator entries of one lane (fragment column n = lane / 4, k = q = lane % 4):
// column n of the interpolation is s = 1 + n/2 + 4 (n&1), column n of the
// divergence Gauss point n/2 + 4 (n&1), so that lane q of a quad owns s = 1+q,
// 5+q and Gauss points q, 4+q.
template <int G, int V> struct MmaOps {
  using C = MmaCfg<G, V>;
  double bm[C::KM > 0 ? C::KM : 1], b0[C::KS > 0 ? C::KS : 1], b1[C::KS > 0 ? C::KS : 1], dm[2], d8[2];
  double dlo[2], dhi[2];  // first and last column of dmx at Gauss points q, 4+q
  __device__ __forceinline__ void load() {
    const int q = threadIdx.x & 3, n = (threadIdx.x & 31) >> 2, kn = (n >> 1) + 4 * (n & 1), sn = 1 + kn;
#pragma unroll
    for (int j = 0; j < C::KM; ++j) bm[j] = (sn <= C::NS && 4 * j + q < G) ? Op<G>::B(sn, 4 * j + q) : 0.0;
#pragma unroll
    for (int k = 0; k < C::KS; ++k) {
      b0[k] = 1 + q <= C::NS ? Op<G>::B(1 + q, 4 * C::KF + k) : 0.0;
      b1[k] = 5 + q <= C::NS ? Op<G>::B(5 + q, 4 * C::KF + k) : 0.0;
    }
#pragma unroll
    for (int j = 0; j < C::NI; ++j) {
      const int s = 1 + 4 * j + q;
      dm[j] = (kn < G && s <= C::NS) ? Op<G>::D(kn, s) : 0.0;
      d8[j] = (G == 9 && n == 0 && s <= C::NS) ? Op<G>::D(G - 1, s) : 0.0;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      dlo[i] = 4 * i + q < G ? Op<G>::D(4 * i + q, 0) : 0.0;
      dhi[i] = 4 * i + q < G ? Op<G>::D(4 * i + q, G) : 0.0;
    }
  }
};

// line (a, b) of row r: across z for direction x (no bank conflicts), else x fastest
template <int G, int D> __device__ __forceinline__ void mma_line(int r, int &a, int &b) {
  if (D == 0) {
    b = r % G;
    a = r / G;
  } else {
    a = r % G;
    b = r / G;
  }
}
template <int G, int D> __device__ __forceinline__ int mma_base(int a, int b) {  // padded Gauss layout
  constexpr int PS = mma_plane(G);
  return D == 0 ? G * a + PS * b : (D == 1 ? a + PS * b : a + G * b);
}
template <int G, int D> __device__ __forceinline__ constexpr int mma_stride() {
  return D == 0 ? 1 : (D == 1 ? G : mma_plane(G));
}

// Where k_vol_mma tests a point's viscosity (vis_flux_x): in the shapes whose register budget takes
// that form better.  Steps, us, without / with the test: p = 6, 125 elements, Smagorinsky's model
// 137.4 / 135.8; p = 7 wide, 64 elements, entropy viscosity 148.7 / 145.7; p = 8, 512 elements, the
// same 574.6 / 566.1 (452 / 404 bytes of spills); the other way round p = 8 wide, 64 elements,
// Smagorinsky's model 200.9 / 202.2, p = 7, 512 elements, the same 337.0 / 341.3, and p = 5.
template <int G, int V>
constexpr bool VIS_TEST = G == 7 || (G == 8 && V == MMA_WIDE) || (G == 9 && V != MMA_WIDE);

// Viscous flux of direction D times gdiag into r from the point's state and its
// 11 interpolated gradient fields (diag_field order).
template <int D, bool MU, bool TEST>
__device__ __forceinline__ void mma_vis(const double *Q, double rr, const double *c, double amu, double gdiag,
                                        const Phys &P, double *r) {
  double Qx[NV], Qy[NV], Qz[NV], fl[NV];
  if (D == 0) {
    Qx[0] = c[0]; Qx[1] = c[1]; Qx[2] = c[2]; Qx[3] = c[3]; Qx[4] = c[4];
    Qy[0] = c[5]; Qy[1] = c[6]; Qy[2] = c[7]; Qy[3] = 0.0; Qy[4] = 0.0;
    Qz[0] = c[8]; Qz[1] = c[9]; Qz[3] = c[10]; Qz[2] = 0.0; Qz[4] = 0.0;
    vis_flux_x<MU, TEST>(Q, rr, Qx, Qy, Qz, amu, P, fl);
  } else if (D == 1) {
    Qy[0] = c[0]; Qy[1] = c[1]; Qy[2] = c[2]; Qy[3] = c[3]; Qy[4] = c[4];
    Qx[0] = c[5]; Qx[1] = c[6]; Qx[2] = c[7]; Qx[3] = 0.0; Qx[4] = 0.0;
    Qz[0] = c[8]; Qz[2] = c[9]; Qz[3] = c[10]; Qz[1] = 0.0; Qz[4] = 0.0;
    vis_flux_y<MU, TEST>(Q, rr, Qx, Qy, Qz, amu, P, fl);
  } else {
    Qz[0] = c[0]; Qz[1] = c[1]; Qz[2] = c[2]; Qz[3] = c[3]; Qz[4] = c[4];
    Qx[0] = c[5]; Qx[1] = c[6]; Qx[3] = c[7]; Qx[2] = 0.0; Qx[4] = 0.0;
    Qy[0] = c[8]; Qy[2] = c[9]; Qy[3] = c[10]; Qy[1] = 0.0; Qy[4] = 0.0;
    vis_flux_z<MU, TEST>(Q, rr, Qx, Qy, Qz, amu, P, fl);
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) r[v] = gdiag * fl[v];
}

// Interpolation to the interior points of a tile's 8 lines: lane r*4+q gets the
// values of line r at s = 1+q (c0) and 5+q (c1).  x: the lane's line at k = q;
// xl: the lane's line at k = 0.
template <int G, int V, int S>
__device__ __forceinline__ void mma_interp(const double *x, const double *xl, const MmaOps<G, V> &O, double &c0,
                                           double &c1) {
  using C = MmaCfg<G, V>;
  c0 = 0.0;
  c1 = 0.0;
#pragma unroll
  for (int j = 0; j < C::KF; ++j) dmma(c0, c1, x[4 * j * S], O.bm[j]);
  if constexpr (C::KM > C::KF) {  // padded k: the line's last value against a zero coefficient
    const int q = threadIdx.x & 3;
    dmma(c0, c1, xl[(4 * C::KF + (q < C::KR ? q : C::KR - 1)) * S], O.bm[C::KF]);
  }
#pragma unroll
  for (int k = 0; k < C::KS; ++k) {
    const double xv = xl[(4 * C::KF + k) * S];
    c0 = __fma_rn(O.b0[k], xv, c0);
    if (C::NI == 2) c1 = __fma_rn(O.b1[k], xv, c1);
  }
}

// Gradients along D of NV1 fields (state sq, from field v0) on a tile's 8 lines: the Lobatto
// lines are interpolated, differentiated and scaled by gmetg(D,D) in registers
// (k_vol's chains); field i goes to out + i * os.
template <int G, int V, int D, int NV1>
__device__ __forceinline__ void mma_grad(int t, const MmaOps<G, V> &O, const double *sq, int v0, const double *QF,
                                         const double *gg, double *out, int os) {
  using C = MmaCfg<G, V>;
  constexpr int L = C::L, G2 = C::G2, NG = C::NG, FS = C::FS;
  constexpr int S = mma_stride<G, D>(), xs = D == 0 ? 1 : (D == 1 ? G : G2);
  const int lane = threadIdx.x & 31, q = lane & 3, n = lane >> 2;
  const bool row = t * 8 + n < G2;
  int a, b;
  mma_line<G, D>(row ? t * 8 + n : G2 - 1, a, b);
  const int pl = mma_base<G, D>(a, b), pq = pl + q * S;
  const double *m = gg + D * NG + gbase<G>(D, a, b) + q * xs;
  const double m0 = q < G ? __ldg(m) : 0.0, m1 = 4 + q < G ? __ldg(m + 4 * xs) : 0.0;
  const double m2 = G == 9 && q == 0 ? __ldg(m + 8 * xs) : 0.0;
  const double *flo = QF + ((face_lo(D) - 1) * 5 + v0) * G2 + a + G * b;
  const double *fhi = QF + ((face_hi(D) - 1) * 5 + v0) * G2 + a + G * b;
  double y0[NV1], y1[NV1];
#pragma unroll
  for (int i = 0; i < NV1; ++i) {
    y0[i] = __ldg(flo + i * G2);
    y1[i] = __ldg(fhi + i * G2);
  }
#pragma unroll
  for (int i = 0; i < NV1; ++i) {
    double c[2];
    mma_interp<G, V, S>(sq + (v0 + i) * FS + pq, sq + (v0 + i) * FS + pl, O, c[0], c[1]);
    double e0 = O.dlo[0] * y0[i], e1 = O.dlo[1] * y0[i], g0 = Op<G>::D(G - 1, 0) * y0[i], g1 = 0.0;
#pragma unroll
    for (int j = 0; j < C::NI; ++j) {
      dmma(e0, e1, c[j], O.dm[j]);
      if (G == 9) dmma(g0, g1, c[j], O.d8[j]);
    }
    e0 = __fma_rn(O.dhi[0], y1[i], e0);
    e1 = __fma_rn(O.dhi[1], y1[i], e1);
    g0 = __fma_rn(Op<G>::D(G - 1, L - 1), y1[i], g0);
    double *o = out + i * os + pq;
    if (row) {
      if (q < G) o[0] = m0 * e0;
      if (4 + q < G) o[4 * S] = m1 * e1;
      if (G == 9 && q == 0) o[8 * S] = m2 * g0;
    }
  }
}

// Adds a direction's part of the divergence to its QTI slot, in the order z (a store), y, x:
// the block barrier between the directions orders the additions, and a reduction at L2
// (rounded to nearest, like the plain sum) needs no load in the tile.
template <int D> __device__ __forceinline__ void mma_add(double *o, double x) {
  if (D == 2)
    *o = x;
  else
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(o), "d"(x) : "memory");
}

// Interior divergence along D (updatea.f90:100-113) of a tile from its lanes' fluxes, k = s - 1:
// lane r*4+q gets line r at Gauss points q and 4+q; the ninth Gauss point of G = 9 is a column
// of its own (q = 0).  qt: the line's first Gauss point.
template <int G, int V, int D>
__device__ __forceinline__ void mma_div(const MmaOps<G, V> &O, const double (&f)[2][NV], bool row, int q, double *qt) {
  using C = MmaCfg<G, V>;
  constexpr int NG = C::NG, xs = D == 0 ? 1 : (D == 1 ? G : C::G2);
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    double e0 = 0.0, e1 = 0.0, g0 = 0.0, g1 = 0.0;
#pragma unroll
    for (int j = 0; j < C::NI; ++j) {
      dmma(e0, e1, f[j][v], O.dm[j]);
      if (G == 9) dmma(g0, g1, f[j][v], O.d8[j]);
    }
    if (row) {
      double *o = qt + v * NG + q * xs;
      if (q < G) mma_add<D>(o, e0);
      if (4 + q < G) mma_add<D>(o + 4 * xs, e1);
      if (G == 9 && q == 0) mma_add<D>(o + 8 * xs, g0);
    }
  }
}

// One tile of direction D: 8 lines, all their interior Lobatto points.  The
// state and gradient fields are interpolated, both fluxes evaluated and the
// interior divergence contracted without leaving the warp's registers.
template <int G, bool MU, int V, int D>
__device__ __forceinline__ void mma_tile(int t, const MmaOps<G, V> &O, const Phys &P, const double *sq, const double *GR, const double *E4,
                                         const double *gm, const double *muhg, const double *nuhg, double *QTI) {
  using C = MmaCfg<G, V>;
  constexpr int G2 = C::G2, NG = C::NG, NL = C::NL, FS = C::FS;
  constexpr int S = mma_stride<G, D>(), xs = D == 0 ? 1 : (D == 1 ? G : G2);
  const int lane = threadIdx.x & 31, q = lane & 3, n = lane >> 2;
  const bool row = t * 8 + n < G2;
  int a, b;
  mma_line<G, D>(row ? t * 8 + n : G2 - 1, a, b);
  const int pl = mma_base<G, D>(a, b), pq = pl + q * S;
  const int l0 = lbase<G>(D, a, b) + (1 + q) * xs;  // Lobatto point s = 1 + q
  double Q[2][NV], c[2][11], gd[2], nu[2] = {0.0, 0.0}, mu[2] = {0.0, 0.0};
  gd[0] = 1 + q <= C::NS ? __ldg(gm + D * NL + l0) : 0.0;
  gd[1] = (C::NI == 2 && 5 + q <= C::NS) ? __ldg(gm + D * NL + l0 + 4 * xs) : 0.0;
#pragma unroll
  for (int v = 0; v < NV; ++v) mma_interp<G, V, S>(sq + v * FS + pq, sq + v * FS + pl, O, Q[0][v], Q[1][v]);
#pragma unroll
  for (int f = 0; f < 11; ++f) {
    const double *x = f == 4 ? E4 : GR + diag_field(D, f) * FS;
    mma_interp<G, V, S>(x + pq, x + pl, O, c[0][f], c[1][f]);
  }
  const bool ev = MU && muhg != nullptr, les = MU && nuhg != nullptr;
  if (ev) {  // EV_Prolong (Prolong_gtol.f90:7-51)
    const double *x = muhg + gbase<G>(D, a, b);
    mma_interp<G, V, xs>(x + q * xs, x, O, mu[0], mu[1]);
  }
  if (les) {  // nut_prolong (staticSmag.f90:206-261): negative values clipped to 0
    const double *x = nuhg + gbase<G>(D, a, b);
    mma_interp<G, V, xs>(x + q * xs, x, O, nu[0], nu[1]);
    if (nu[0] < 0.0) nu[0] = 0.0;
    if (nu[1] < 0.0) nu[1] = 0.0;
  }
  double f[2][NV];
#pragma unroll
  for (int i = 0; i < C::NI; ++i) {
    double amu = 1.0;  // Vis_Fluxes_new.f90:123-125
    if (les) amu = amu + nu[i] * Q[i][0];
    if (ev) amu = amu + mu[i];
    const double rr = 1.0 / Q[i][0];
    double r[NV], fi[NV];
    mma_vis<D, MU, VIS_TEST<G, V>>(Q[i], rr, c[i], amu, gd[i], P, r);
    euler_flux(D, Q[i], rr, P.gm1, fi);
    const bool in = (i == 0 ? 1 : 5) + q <= C::NS;  // padded points contribute exact zeros
#pragma unroll
    for (int v = 0; v < NV; ++v) f[i][v] = in ? gd[i] * fi[v] - ddiv(r[v], P.re, P.r_re) : 0.0;
  }
  mma_div<G, V, D>(O, f, row, q, QTI + gbase<G>(D, a, b));
}

// Viscous fluxes at both face points of one line of direction D per lane
// (Vis_Fluxes_new.f90:115-228), written to VF.
template <int G, bool MU, int V, int D>
__device__ __forceinline__ void mma_faces(int ln, const Phys &P, const double *QF, const double *GR, const double *E4,
                                          const double *gm, const double *muhg, const double *nuhg, double *VF) {
  using C = MmaCfg<G, V>;
  constexpr int L = C::L, G2 = C::G2, NL = C::NL, FS = C::FS;
  constexpr int S = mma_stride<G, D>(), xs = D == 0 ? 1 : (D == 1 ? G : G2);
  const int a = ln % G, b = ln / G;
  const int pl = mma_base<G, D>(a, b);
  const double *qlo = QF + (face_lo(D) - 1) * 5 * G2 + ln, *qhi = QF + (face_hi(D) - 1) * 5 * G2 + ln;
  const double *g = gm + D * NL + lbase<G>(D, a, b);
  double Q[2][NV], gd[2] = {__ldg(g), __ldg(g + (L - 1) * xs)};
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    Q[0][v] = __ldg(qlo + v * G2);
    Q[1][v] = __ldg(qhi + v * G2);
  }
  double c[2][11], nu[2] = {0.0, 0.0}, mu[2] = {0.0, 0.0};
  auto ends = [&](const double *x, int st, double &lo, double &hi) {
    const double x0 = x[0];
    lo = Op<G>::B(0, 0) * x0;
    hi = Op<G>::B(L - 1, 0) * x0;
#pragma unroll
    for (int k = 1; k < G; ++k) {
      const double xv = x[k * st];
      lo = __fma_rn(Op<G>::B(0, k), xv, lo);
      hi = __fma_rn(Op<G>::B(L - 1, k), xv, hi);
    }
  };
#pragma unroll
  for (int f = 0; f < 11; ++f) ends((f == 4 ? E4 : GR + diag_field(D, f) * FS) + pl, S, c[0][f], c[1][f]);
  const bool ev = MU && muhg != nullptr, les = MU && nuhg != nullptr;
  if (ev) ends(muhg + gbase<G>(D, a, b), xs, mu[0], mu[1]);
  if (les) {
    ends(nuhg + gbase<G>(D, a, b), xs, nu[0], nu[1]);
    if (nu[0] < 0.0) nu[0] = 0.0;
    if (nu[1] < 0.0) nu[1] = 0.0;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    double r[NV];
    double amu = 1.0;
    if (les) amu = amu + nu[i] * Q[i][0];
    if (ev) amu = amu + mu[i];
    mma_vis<D, MU, VIS_TEST<G, V>>(Q[i], 1.0 / Q[i][0], c[i], amu, gd[i], P, r);
    double *o = VF + ((i ? face_hi(D) : face_lo(D)) - 1) * 5 * G2 + ln;
#pragma unroll
    for (int v = 0; v < NV; ++v) o[v * G2] = r[v];
  }
}

// Phase of direction D: its face points, the energy gradient of the next
// direction (z, y, x), and its tiles, drawn by the warps from one list.
template <int G, bool MU, int V, int D>
__device__ __forceinline__ void mma_phase(int *next, const MmaOps<G, V> &O, const Phys &P, const double *sq, const double *GR, const double *E4,
                                          double *E4n, const double *QF, const double *gg, const double *gm,
                                          const double *muhg, const double *nuhg, double *VF, double *QTI) {
  using C = MmaCfg<G, V>;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int i = C::NW - 1 - w; i < C::NLW; i += C::NW)
    if (i * 32 + lane < C::G2) mma_faces<G, MU, V, D>(i * 32 + lane, P, QF, GR, E4, gm, muhg, nuhg, VF);
  __syncwarp();
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(next, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= (D > 0 ? 2 : 1) * C::NTILE) break;
    if (t >= C::NTILE)  // the next direction's energy gradient (needed on grid D only)
      mma_grad<G, V, (D > 0 ? D - 1 : 0), 1>(t - C::NTILE, O, sq, 4, QF, gg, E4n, 0);
    else
      mma_tile<G, MU, V, D>(t, O, P, sq, GR, E4, gm, muhg, nuhg, QTI);
  }
}

// Temperature gradient along D (EV runs, SAVE == 2): the five Lobatto lines, the
// temperature on them (RHS.f90:66-83), its derivative scaled by gmetg(D,D) (GEN: by
// gmetg(D,c), added to the three components in the order of the directions).
template <int G, int V, int D, bool GEN = false>
__device__ __forceinline__ void mma_tgrad(int ln, const double *sq, const double *QF, const double *gg, double *EVB,
                                          double gamma) {
  constexpr int L = G + 1, G2 = G * G, NG = G * G * G, FS = MmaCfg<G, V>::FS;
  constexpr int S = mma_stride<G, D>(), xs = D == 0 ? 1 : (D == 1 ? G : G2);
  const int a = ln % G, b = ln / G;
  const int pl = mma_base<G, D>(a, b), p0 = gbase<G>(D, a, b);
  double y[5][L];
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    double x[G];
#pragma unroll
    for (int kk = 0; kk < G; ++kk) x[kk] = sq[v * FS + pl + kk * S];
    y[v][0] = __ldg(QF + (face_lo(D) - 1) * 5 * G2 + v * G2 + ln);
    y[v][L - 1] = __ldg(QF + (face_hi(D) - 1) * 5 * G2 + v * G2 + ln);
#pragma unroll
    for (int s = 1; s < L - 1; ++s) {
      double acc = Op<G>::B(s, 0) * x[0];
#pragma unroll
      for (int kk = 1; kk < G; ++kk) acc = __fma_rn(Op<G>::B(s, kk), x[kk], acc);
      y[v][s] = acc;
    }
  }
  double T[L];
#pragma unroll
  for (int s = 0; s < L; ++s) {
    const double q1 = y[0][s], q2 = y[1][s], q3 = y[2][s], q4 = y[3][s], q5 = y[4][s];
    const double r1 = 1.0 / q1, u = ddiv(q2, q1, r1), v = ddiv(q3, q1, r1), w = ddiv(q4, q1, r1);
    const double Pp = (gamma - 1.0) * (q5 - 0.5 * q1 * (u * u + v * v + w * w));
    T[s] = ddiv(Pp * gamma, q1, r1);
  }
#pragma unroll
  for (int kk = 0; kk < G; ++kk) {
    double acc = Op<G>::D(kk, 0) * T[0];
#pragma unroll
    for (int s = 1; s < L; ++s) acc = __fma_rn(Op<G>::D(kk, s), T[s], acc);
    const int p = p0 + kk * xs;
    if (GEN) {  // contributions of direction D to the three components
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double val = gg[p * 9 + D + 3 * c] * acc;
        EVB[(12 + c) * NG + p] = D == 0 ? val : EVB[(12 + c) * NG + p] + val;
      }
    } else {
      EVB[(12 + D) * NG + p] = gg[D * NG + p] * acc;
    }
  }
}

// Q*jacob (fluxesH_newa.f90:262-272) into the padded state, all of a thread's loads in flight
// at once.
template <int G, int NT> __device__ __forceinline__ void mma_load(const double *JQ, const double *jac, double *sq) {
  constexpr int G2 = G * G, NG = G * G * G, PS = mma_plane(G), NQ = (5 * NG + NT - 1) / NT;
  const int tid = threadIdx.x;
  double qv[NQ], jv[NQ];
#pragma unroll
  for (int j = 0; j < NQ; ++j) {
    const int i = tid + j * NT;
    if (i < 5 * NG) {
      qv[j] = JQ[i];
      jv[j] = jac[i % NG];
    }
  }
#pragma unroll
  for (int j = 0; j < NQ; ++j) {
    const int i = tid + j * NT;
    if (i < 5 * NG) sq[i / G2 * PS + i % G2] = qv[j] * jv[j];
  }
}

template <int G, bool MU, int SAVE, int V = 0>
__global__ void __launch_bounds__(MmaCfg<G, V>::NT, MmaCfg<G, V>::MINB) k_vol_mma(VolArgs A) {
  using C = MmaCfg<G, V>;
  constexpr int G2 = C::G2, NG = C::NG, NL = C::NL, NT = C::NT, FS = C::FS, PS = C::PS;
  extern __shared__ double sm[];
  double *sq = sm;              // [5] state
  double *GR = sq + 5 * FS;     // [12] Gauss gradients, field v*3 + direction
  double *E0 = GR + 12 * FS;    // energy gradient along z, then along x
  double *E1 = E0 + FS;         // energy gradient along y
  int *next = reinterpret_cast<int *>(E1 + FS);  // [3] work lists of the phases
  const int tid = threadIdx.x, k = blockIdx.x;
  const double *JQ = A.JQ + (long long)k * A.sq;
  const double *jac = A.jac + (long long)k * NG;
  const double *QF = A.QF + (long long)k * 30 * G2;
  double *VF = A.VF + (long long)k * 30 * G2;
  const double *gg = A.gg + (long long)k * 3 * NG;
  const double *gm = A.gm + (long long)k * 3 * NL;
  const double *muhg = MU && A.muhg ? A.muhg + (long long)k * NG : nullptr;  // viscosity models in use
  const double *nuhg = MU && A.nuhg ? A.nuhg + (long long)k * NG : nullptr;
  double *EVB = SAVE ? A.EVB + (long long)k * 15 * NG : nullptr;
  double *QTI = A.QTI + (long long)k * 5 * NG;
  Phys P = A.P;
  if (A.rec) {  // per-case Reynolds number
    const int cs = A.ecase[k];
    P.re = A.rec[2 * cs];
    P.r_re = A.rec[2 * cs + 1];
  }
  if (tid == 0) {
    prefetch_l2_bulk(gg, 3 * NG);
    prefetch_l2_bulk(gm, 3 * NL);
    prefetch_l2_bulk(QF, 30 * G2);
    if (muhg) prefetch_l2_bulk(muhg, NG);
    if (nuhg) prefetch_l2_bulk(nuhg, NG);
  }
  if (tid < 3) next[tid] = 0;
  long long t_ph_ = 0;
#ifdef DSEM_PHASE_TIMING
  t_ph_ = clock64();
#endif
  mma_load<G, NT>(JQ, jac, sq);
  __syncthreads();
  PHASE_MARK(0);
  MmaOps<G, V> O;
  O.load();
  // pass 1: Gauss gradients of fields 0..3 (and of the energy along z), a tile of lines per task
  for (int t = tid >> 5; t < 3 * C::NTILE; t += C::NW) {
    if (t < C::NTILE) {
      mma_grad<G, V, 2, 4>(t, O, sq, 0, QF, gg, GR + 2 * FS, 3 * FS);
      mma_grad<G, V, 2, 1>(t, O, sq, 4, QF, gg, E0, 0);
    } else if (t < 2 * C::NTILE) {
      mma_grad<G, V, 1, 4>(t - C::NTILE, O, sq, 0, QF, gg, GR + FS, 3 * FS);
    } else {
      mma_grad<G, V, 0, 4>(t - 2 * C::NTILE, O, sq, 0, QF, gg, GR, 3 * FS);
    }
  }
  if (SAVE == 2) {
    for (int t = tid; t < 3 * G2; t += NT) {
      const int D = t / G2, ln = t - D * G2;
      if (D == 0)
        mma_tgrad<G, V, 0>(ln, sq, QF, gg, EVB, P.gamma);
      else if (D == 1)
        mma_tgrad<G, V, 1>(ln, sq, QF, gg, EVB, P.gamma);
      else
        mma_tgrad<G, V, 2>(ln, sq, QF, gg, EVB, P.gamma);
    }
  }
  __syncthreads();
  PHASE_MARK(1);
  if (SAVE) {
    for (int i = tid; i < 12 * NG; i += NT) EVB[i] = GR[i / G2 * PS + i % G2];
  }
  // pass 2: z, y, x
  mma_phase<G, MU, V, 2>(next + 0, O, P, sq, GR, E0, E1, QF, gg, gm, muhg, nuhg, VF, QTI);
  __syncthreads();
  PHASE_MARK(2);
  mma_phase<G, MU, V, 1>(next + 1, O, P, sq, GR, E1, E0, QF, gg, gm, muhg, nuhg, VF, QTI);
  __syncthreads();
  PHASE_MARK(3);
  mma_phase<G, MU, V, 0>(next + 2, O, P, sq, GR, E0, E1, QF, gg, gm, muhg, nuhg, VF, QTI);
  PHASE_MARK(4);
}

// ------------------------------------------------------------ general metrics
// k_vol_mma_gen: the same for elements with full metrics (rotated, skewed or curved), all
// 15 gradient components kept (k_vol's sums over the directions x, y, z) and all three
// fluxes formed at every point.  Bound by the FP64 pipe like the diagonal kernel, with about
// twice its work.  20 shared fields: two elements fit an SM's shared memory at p = 7 (87 KB
// each), one at p = 8 (121 KB); the 12 warps of 168 registers take one element per SM at both.  Measured, ms per volume launch, k_vol -> this: 10^3 curved
// elements of p = 8 0.414 -> 0.217, p = 7 0.252 -> 0.135, 12^3 of p = 6 0.280 -> 0.169,
// p = 5 0.168 -> 0.124, 14^3 of p = 4 0.212 -> 0.096, p = 3 0.090 -> 0.047.

// Contributions of the derivative along D to the Gauss gradients of the five fields on a
// tile's lines (Gauss_Deriv, SolnDerivsc.f90:36-80): stored for D = 0, added after.
template <int G, int V, int D>
__device__ __forceinline__ void mma_gen_grad(int t, const MmaOps<G, V> &O, const double *sq, const double *QF,
                                             const double *gg, double *GR) {
  using C = MmaCfg<G, V>;
  constexpr int L = C::L, G2 = C::G2, FS = C::FS;
  constexpr int S = mma_stride<G, D>(), xs = D == 0 ? 1 : (D == 1 ? G : G2);
  const int lane = threadIdx.x & 31, q = lane & 3, n = lane >> 2;
  const bool row = t * 8 + n < G2;
  int a, b;
  mma_line<G, D>(row ? t * 8 + n : G2 - 1, a, b);
  const int pl = mma_base<G, D>(a, b), pq = pl + q * S;
  const double *m = gg + (gbase<G>(D, a, b) + q * xs) * 9 + D;
  double mt[3][3];  // [Gauss point q, 4+q, 8][component]
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const bool in = i == 0 ? q < G : (i == 1 ? 4 + q < G : G == 9 && q == 0);
#pragma unroll
    for (int c = 0; c < 3; ++c) mt[i][c] = in ? __ldg(m + 4 * i * xs * 9 + 3 * c) : 0.0;
  }
  const double *flo = QF + (face_lo(D) - 1) * 5 * G2 + a + G * b, *fhi = QF + (face_hi(D) - 1) * 5 * G2 + a + G * b;
  double y0[NV], y1[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    y0[v] = __ldg(flo + v * G2);
    y1[v] = __ldg(fhi + v * G2);
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    double c[2];
    mma_interp<G, V, S>(sq + v * FS + pq, sq + v * FS + pl, O, c[0], c[1]);
    double w[3] = {O.dlo[0] * y0[v], O.dlo[1] * y0[v], Op<G>::D(G - 1, 0) * y0[v]}, g1 = 0.0;
#pragma unroll
    for (int j = 0; j < C::NI; ++j) {
      dmma(w[0], w[1], c[j], O.dm[j]);
      if (G == 9) dmma(w[2], g1, c[j], O.d8[j]);
    }
    w[0] = __fma_rn(O.dhi[0], y1[v], w[0]);
    w[1] = __fma_rn(O.dhi[1], y1[v], w[1]);
    w[2] = __fma_rn(Op<G>::D(G - 1, L - 1), y1[v], w[2]);
    if (row) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const bool in = i == 0 ? q < G : (i == 1 ? 4 + q < G : G == 9 && q == 0);
        if (!in) continue;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          double *o = GR + (v * 3 + k) * FS + pq + 4 * i * S;
          const double val = mt[i][k] * w[i];
          *o = D == 0 ? val : *o + val;
        }
      }
    }
  }
}

// r = m . (viscous fluxes), and with INV also e = m . (Euler fluxes) at one point.
template <bool INV, bool MU>
__device__ __forceinline__ void mma_gen_flux(const double *Q, const double *c, const double *m, double amu,
                                             const Phys &P, double *r, double *e) {
  double Qx[NV], Qy[NV], Qz[NV], f[NV], g[NV], h[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    Qx[v] = c[v * 3];
    Qy[v] = c[v * 3 + 1];
    Qz[v] = c[v * 3 + 2];
  }
  const double rr = 1.0 / Q[0];
  vis_flux_x<MU>(Q, rr, Qx, Qy, Qz, amu, P, f);
  vis_flux_y<MU>(Q, rr, Qx, Qy, Qz, amu, P, g);
  vis_flux_z<MU>(Q, rr, Qx, Qy, Qz, amu, P, h);
#pragma unroll
  for (int v = 0; v < NV; ++v) r[v] = m[0] * f[v] + m[1] * g[v] + m[2] * h[v];
  if (INV) {
    euler_fluxes3(Q, rr, P.gm1, f, g, h);
#pragma unroll
    for (int v = 0; v < NV; ++v) e[v] = m[0] * f[v] + m[1] * g[v] + m[2] * h[v];
  }
}

// One tile of direction D (mma_tile with full metrics).
template <int G, bool MU, int V, int D>
__device__ __forceinline__ void mma_gen_tile(int t, const MmaOps<G, V> &O, const Phys &P, const double *sq,
                                             const double *GR, const double *gm, const double *muhg, double *QTI) {
  using C = MmaCfg<G, V>;
  constexpr int G2 = C::G2, NG = C::NG, NL = C::NL, FS = C::FS;
  constexpr int S = mma_stride<G, D>(), xs = D == 0 ? 1 : (D == 1 ? G : G2);
  const int lane = threadIdx.x & 31, q = lane & 3, n = lane >> 2;
  const bool row = t * 8 + n < G2;
  int a, b;
  mma_line<G, D>(row ? t * 8 + n : G2 - 1, a, b);
  const int pl = mma_base<G, D>(a, b), pq = pl + q * S;
  const double *g3 = gm + ((long long)D * NL + lbase<G>(D, a, b) + (1 + q) * xs) * 3;
  double m[2][3], Q[2][NV], c[2][15], mu[2] = {0.0, 0.0}, f[2][NV];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const bool in = i < C::NI && (i == 0 ? 1 : 5) + q <= C::NS;
#pragma unroll
    for (int k = 0; k < 3; ++k) m[i][k] = in ? __ldg(g3 + i * 12 * xs + k) : 0.0;
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) mma_interp<G, V, S>(sq + v * FS + pq, sq + v * FS + pl, O, Q[0][v], Q[1][v]);
#pragma unroll
  for (int j = 0; j < 15; ++j) mma_interp<G, V, S>(GR + j * FS + pq, GR + j * FS + pl, O, c[0][j], c[1][j]);
  if (MU) {  // EV_Prolong (Prolong_gtol.f90:7-51)
    const double *x = muhg + gbase<G>(D, a, b);
    mma_interp<G, V, xs>(x + q * xs, x, O, mu[0], mu[1]);
  }
#pragma unroll
  for (int i = 0; i < C::NI; ++i) {
    double amu = 1.0, r[NV], e[NV];
    if (MU) amu = amu + mu[i];
    mma_gen_flux<true, MU>(Q[i], c[i], m[i], amu, P, r, e);
    const bool in = (i == 0 ? 1 : 5) + q <= C::NS;
#pragma unroll
    for (int v = 0; v < NV; ++v) f[i][v] = in ? e[v] - ddiv(r[v], P.re, P.r_re) : 0.0;
  }
  mma_div<G, V, D>(O, f, row, q, QTI + gbase<G>(D, a, b));
}

// Viscous flux at one face point of a line of direction D per lane (END 0 low, 1 high).
template <int G, bool MU, int V, int D, int END>
__device__ __forceinline__ void mma_gen_face(int ln, const Phys &P, const double *QF, const double *GR,
                                             const double *gm, const double *muhg, double *VF) {
  using C = MmaCfg<G, V>;
  constexpr int L = C::L, G2 = C::G2, NL = C::NL, FS = C::FS, s = END ? L - 1 : 0;
  constexpr int S = mma_stride<G, D>(), xs = D == 0 ? 1 : (D == 1 ? G : G2);
  const int a = ln % G, b = ln / G, pl = mma_base<G, D>(a, b);
  const int o = ((END ? face_hi(D) : face_lo(D)) - 1) * 5 * G2 + ln;
  const double *g3 = gm + ((long long)D * NL + lbase<G>(D, a, b) + s * xs) * 3;
  double Q[NV], m[3], c[15], r[NV];
#pragma unroll
  for (int k = 0; k < 3; ++k) m[k] = __ldg(g3 + k);
#pragma unroll
  for (int v = 0; v < NV; ++v) Q[v] = __ldg(QF + o + v * G2);
  auto end = [&](const double *x, int st) {
    double acc = Op<G>::B(s, 0) * x[0];
#pragma unroll
    for (int k = 1; k < G; ++k) acc = __fma_rn(Op<G>::B(s, k), x[k * st], acc);
    return acc;
  };
#pragma unroll
  for (int j = 0; j < 15; ++j) c[j] = end(GR + j * FS + pl, S);
  double amu = 1.0;
  if (MU) amu = amu + end(muhg + gbase<G>(D, a, b), xs);
  mma_gen_flux<false, MU>(Q, c, m, amu, P, r, nullptr);
#pragma unroll
  for (int v = 0; v < NV; ++v) VF[o + v * G2] = r[v];
}

template <int G, bool MU, int V, int D>
__device__ __forceinline__ void mma_gen_phase(int *next, const MmaOps<G, V> &O, const Phys &P, const double *sq,
                                              const double *GR, const double *QF, const double *gm,
                                              const double *muhg, double *VF, double *QTI) {
  using C = MmaCfg<G, V>;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int i = C::NW - 1 - w; i < 2 * C::NLW; i += C::NW) {
    const int ln = (i >> 1) * 32 + lane;
    if (ln >= C::G2) continue;
    if (i & 1)
      mma_gen_face<G, MU, V, D, 1>(ln, P, QF, GR, gm, muhg, VF);
    else
      mma_gen_face<G, MU, V, D, 0>(ln, P, QF, GR, gm, muhg, VF);
  }
  __syncwarp();
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(next, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= C::NTILE) break;
    mma_gen_tile<G, MU, V, D>(t, O, P, sq, GR, gm, muhg, QTI);
  }
}

template <int G, bool MU, int SAVE, int V = MMA_GEN>
__global__ void __launch_bounds__(MmaCfg<G, V>::NT, MmaCfg<G, V>::MINB) k_vol_mma_gen(VolArgs A) {
  using C = MmaCfg<G, V>;
  constexpr int G2 = C::G2, NG = C::NG, NL = C::NL, NT = C::NT, FS = C::FS, PS = C::PS;
  extern __shared__ double sm[];
  double *sq = sm;            // [5] state
  double *GR = sq + 5 * FS;   // [15] Gauss gradients, field v*3 + component
  int *next = reinterpret_cast<int *>(GR + 15 * FS);
  const int tid = threadIdx.x, k = blockIdx.x;
  const double *JQ = A.JQ + (long long)k * A.sq;
  const double *jac = A.jac + (long long)k * NG;
  const double *QF = A.QF + (long long)k * 30 * G2;
  double *VF = A.VF + (long long)k * 30 * G2;
  const double *gg = A.gg + (long long)k * 9 * NG;
  const double *gm = A.gm + (long long)k * 9 * NL;
  const double *muhg = MU ? A.muhg + (long long)k * NG : nullptr;
  double *EVB = SAVE ? A.EVB + (long long)k * 15 * NG : nullptr;
  double *QTI = A.QTI + (long long)k * 5 * NG;
  Phys P = A.P;
  if (A.rec) {  // per-case Reynolds number
    const int cs = A.ecase[k];
    P.re = A.rec[2 * cs];
    P.r_re = A.rec[2 * cs + 1];
  }
  if (tid == 0) {
    prefetch_l2_bulk(gg, 9 * NG);
    prefetch_l2_bulk(gm, 9 * NL);
    prefetch_l2_bulk(QF, 30 * G2);
    if (MU) prefetch_l2_bulk(muhg, NG);
  }
  if (tid < 3) next[tid] = 0;
  mma_load<G, NT>(JQ, jac, sq);
  MmaOps<G, V> O;
  O.load();
  __syncthreads();
  // pass 1: Gauss gradients, the directions' contributions added in the order x, y, z
  for (int t = tid >> 5; t < C::NTILE; t += C::NW) mma_gen_grad<G, V, 0>(t, O, sq, QF, gg, GR);
  if (SAVE == 2)
    for (int t = tid; t < G2; t += NT) mma_tgrad<G, V, 0, true>(t, sq, QF, gg, EVB, P.gamma);
  __syncthreads();
  for (int t = tid >> 5; t < C::NTILE; t += C::NW) mma_gen_grad<G, V, 1>(t, O, sq, QF, gg, GR);
  if (SAVE == 2)
    for (int t = tid; t < G2; t += NT) mma_tgrad<G, V, 1, true>(t, sq, QF, gg, EVB, P.gamma);
  __syncthreads();
  for (int t = tid >> 5; t < C::NTILE; t += C::NW) mma_gen_grad<G, V, 2>(t, O, sq, QF, gg, GR);
  if (SAVE == 2)
    for (int t = tid; t < G2; t += NT) mma_tgrad<G, V, 2, true>(t, sq, QF, gg, EVB, P.gamma);
  __syncthreads();
  if (SAVE) {
    for (int i = tid; i < 12 * NG; i += NT) EVB[i] = GR[i / G2 * PS + i % G2];
  }
  // pass 2: z, y, x
  mma_gen_phase<G, MU, V, 2>(next + 0, O, P, sq, GR, QF, gm, muhg, VF, QTI);
  __syncthreads();
  mma_gen_phase<G, MU, V, 1>(next + 1, O, P, sq, GR, QF, gm, muhg, VF, QTI);
  __syncthreads();
  mma_gen_phase<G, MU, V, 0>(next + 2, O, P, sq, GR, QF, gm, muhg, VF, QTI);
}

}  // namespace dsem
