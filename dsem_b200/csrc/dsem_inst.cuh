// dsem_inst.cuh -- definitions of Launch<G>; included once per order by inst_g*.cu.
#pragma once
#include "dsem_launch.h"
#include "dsem_stage.cuh"
#include "dsem_vol_diag.cuh"
#include "dsem_vol_mma.cuh"
#include "dsem_lobatto.cuh"

namespace dsem {

template <int G> cudaError_t Launch<G>::set_ops(const double *h, int n) {
  if (n != OPS_TOTAL) return cudaErrorInvalidValue;
  return cudaMemcpyToSymbol(c_ops, h, sizeof(double) * OPS_TOTAL);
}

// general metrics, p = 1, 2, and small launches at p = 4, 5
template <int G, bool EV, int SAVE> static cudaError_t vol_one(const VolArgs &a, int nel, cudaStream_t s) {
  using C = VolCfg<G, EV>;
  auto kern = k_vol<G, EV, SAVE>;
  static std::atomic<unsigned long long> attr{0};
  cudaError_t e = set_smem_once(kern, C::SMEM, attr);
  if (e != cudaSuccess) return e;
  if (nel <= 0 || !a.JQ) return cudaSuccess;
  kern<<<nel, C::NT, C::SMEM, s>>>(a);
  return cudaGetLastError();
}

// diagonal metrics, p = 1, 2
template <int G, bool EV, int SAVE> static cudaError_t vol_diag_one(const VolArgs &a, int nel, cudaStream_t s) {
  using C = VolDiagCfg<G>;
  auto kern = k_vol_diag<G, EV, SAVE>;
  static std::atomic<unsigned long long> attr{0};
  cudaError_t e = set_smem_once(kern, C::SMEM, attr);
  if (e != cudaSuccess) return e;
  if (nel <= 0 || !a.JQ) return cudaSuccess;
  kern<<<nel, C::NT, C::SMEM, s>>>(a);
  return cudaGetLastError();
}

// diagonal metrics, p >= 3: line contractions on the FP64 matrix instruction
template <int G, bool MU, int SAVE, int V = 0>
static cudaError_t vol_mma_one(const VolArgs &a, int nel, cudaStream_t s) {
  using C = MmaCfg<G, V>;
  auto kern = k_vol_mma<G, MU, SAVE, V>;
  static std::atomic<unsigned long long> attr{0};
  cudaError_t e = set_smem_once(kern, C::SMEM, attr);
  if (e != cudaSuccess) return e;
  if (nel <= 0 || !a.JQ) return cudaSuccess;
  kern<<<nel, C::NT, C::SMEM, s>>>(a);
  return cudaGetLastError();
}

// general metrics, p >= 3
template <int G, bool MU, int SAVE, int V = MMA_GEN>
static cudaError_t vol_gen_one(const VolArgs &a, int nel, cudaStream_t s) {
  using C = MmaCfg<G, V>;
  auto kern = k_vol_mma_gen<G, MU, SAVE, V>;
  static std::atomic<unsigned long long> attr{0};
  cudaError_t e = set_smem_once(kern, C::SMEM, attr);
  if (e != cudaSuccess) return e;
  if (nel <= 0 || !a.JQ) return cudaSuccess;
  kern<<<nel, C::NT, C::SMEM, s>>>(a);
  return cudaGetLastError();
}

// MU: with a viscosity model (entropy viscosity, Smagorinsky).  Entropy viscosity always saves the
// temperature gradient too (SAVE = 2) and takes no explicit shape, but the default rule's shape 3 at p = 4.
template <int G, bool MU, int SAVE> static cudaError_t vol_mma_shape(const VolArgs &a, int nel, cudaStream_t s, int v) {
  if constexpr (vol_has_variants(G) && SAVE != 2) {
    switch (v) {
      case 1: return vol_mma_one<G, MU, SAVE, 1>(a, nel, s);
      case 2: return vol_mma_one<G, MU, SAVE, 2>(a, nel, s);
      case 3: return vol_mma_one<G, MU, SAVE, 3>(a, nel, s);
      case 4: return vol_mma_one<G, MU, SAVE, 4>(a, nel, s);
    }
  }
  if constexpr (G == 5 && SAVE == 2)
    if (v == 3) return vol_mma_one<G, MU, SAVE, 3>(a, nel, s);
  return v == MMA_WIDE ? vol_mma_one<G, MU, SAVE, MMA_WIDE>(a, nel, s) : vol_mma_one<G, MU, SAVE>(a, nel, s);
}
template <int G, bool MU, int SAVE> static cudaError_t vol_gen_shape(const VolArgs &a, int nel, cudaStream_t s, int v) {
  if constexpr (G < 8)
    if (v == MMA_GEN_WIDE) return vol_gen_one<G, MU, SAVE, MMA_GEN_WIDE>(a, nel, s);
  return vol_gen_one<G, MU, SAVE>(a, nel, s);
}

template <int G>
cudaError_t Launch<G>::vol(const VolArgs &a, int nel, bool diag, int mode, cudaStream_t s, int variant) {
  const bool ev = mode == VOL_EV || mode == VOL_EV_SAVE;
  if constexpr (G >= 4) {
    const int v = vol_shape(G, diag, nel, ev, variant);
    if (diag) {
      VolArgs b = a;
      if (!ev) b.muhg = nullptr;
      if (ev || a.nuhg) switch (mode) {
          case VOL_SAVE: return vol_mma_shape<G, true, 1>(b, nel, s, v);
          case VOL_EV_SAVE: return vol_mma_shape<G, true, 2>(b, nel, s, v);
          default: return vol_mma_shape<G, true, 0>(b, nel, s, v);
        }
      return mode == VOL_SAVE ? vol_mma_shape<G, false, 1>(b, nel, s, v) : vol_mma_shape<G, false, 0>(b, nel, s, v);
    }
    if constexpr (vol_point_max(G) > 0)
      if (v == VOL_POINT) switch (mode) {
          case VOL_SAVE: return vol_one<G, false, 1>(a, nel, s);
          case VOL_EV: return vol_one<G, true, 0>(a, nel, s);
          case VOL_EV_SAVE: return vol_one<G, true, 2>(a, nel, s);
          default: return vol_one<G, false, 0>(a, nel, s);
        }
    switch (mode) {
      case VOL_SAVE: return vol_gen_shape<G, false, 1>(a, nel, s, v);
      case VOL_EV: return vol_gen_shape<G, true, 0>(a, nel, s, v);
      case VOL_EV_SAVE: return vol_gen_shape<G, true, 2>(a, nel, s, v);
      default: return vol_gen_shape<G, false, 0>(a, nel, s, v);
    }
  } else if (diag) {
    switch (mode) {
      case VOL_SAVE: return vol_diag_one<G, false, 1>(a, nel, s);
      case VOL_EV: return vol_diag_one<G, true, 0>(a, nel, s);
      case VOL_EV_SAVE: return vol_diag_one<G, true, 2>(a, nel, s);
      default: return vol_diag_one<G, false, 0>(a, nel, s);
    }
  } else {
    switch (mode) {
      case VOL_SAVE: return vol_one<G, false, 1>(a, nel, s);
      case VOL_EV: return vol_one<G, true, 0>(a, nel, s);
      case VOL_EV_SAVE: return vol_one<G, true, 2>(a, nel, s);
      default: return vol_one<G, false, 0>(a, nel, s);
    }
  }
}

template <int G> cudaError_t Launch<G>::update(const UpdArgs &a, int nel, cudaStream_t s) {
  constexpr size_t smem = UPD_SMEM<G>;
  static_assert(smem <= 48 * 1024, "more needs the kernel's shared-memory attribute");
  if (nel <= 0) return cudaSuccess;
  if (a.fmc)
    k_update<G, true><<<nel, 256, smem, s>>>(a);
  else
    k_update<G, false><<<nel, 256, smem, s>>>(a);
  return cudaGetLastError();
}

template <int G> cudaError_t Launch<G>::trace(const TraceArgs &a, int nel, cudaStream_t s) {
  if (nel <= 0) return cudaSuccess;
  k_trace<G><<<nel, 256, sizeof(double) * 5 * G * G * G, s>>>(a);
  return cudaGetLastError();
}

template <int G> cudaError_t Launch<G>::lob_keep(const LobArgs &a, int nel, cudaStream_t s) {
  if (nel <= 0) return cudaSuccess;
  k_lob_keep<G><<<nel, 256, sizeof(double) * 5 * G * G * G, s>>>(a);
  return cudaGetLastError();
}

template <int G> cudaError_t Launch<G>::lob_grad(const LobArgs &a, int nel, bool diag, cudaStream_t s) {
  if (nel <= 0) return cudaSuccess;
  if (diag)
    k_lob_grad<G, true><<<nel, 256, 0, s>>>(a);
  else
    k_lob_grad<G, false><<<nel, 256, 0, s>>>(a);
  return cudaGetLastError();
}

template <int G> cudaError_t Launch<G>::ev(const EvArgs &a, int nel, cudaStream_t s) {
  if (nel <= 0) return cudaSuccess;
  k_ev<G><<<nel, 256, 0, s>>>(a);
  return cudaGetLastError();
}

template <int G> cudaError_t Launch<G>::les(const LesArgs &a, int nel, cudaStream_t s) {
  if (nel <= 0) return cudaSuccess;
  k_les<G><<<nel, 128, 0, s>>>(a);
  return cudaGetLastError();
}

template <int G>
cudaError_t Launch<G>::face_inv(const MortarC *mc, int nm, double *QF, double *FF, const double *nh, const double *nrm,
                                double gamma, cudaStream_t s) {
  if (nm <= 0) return cudaSuccess;
  const long long n = (long long)nm * G * G;
  k_face_inv<G><<<(unsigned)((n + 127) / 128), 128, 0, s>>>(mc, nm, QF, FF, nh, nrm, RoeC::of(gamma));
  return cudaGetLastError();
}

template <int G>
cudaError_t Launch<G>::face_inv_from(const MortarC *mc, int nm, const double *QFR, double *QF, double *FF,
                                     const double *nh, const double *nrm, double gamma, cudaStream_t s) {
  if (nm <= 0) return cudaSuccess;
  const long long n = (long long)nm * G * G;
  k_face_inv_from<G><<<(unsigned)((n + 127) / 128), 128, 0, s>>>(mc, nm, QFR, QF, FF, nh, nrm, RoeC::of(gamma));
  return cudaGetLastError();
}

template <int G> cudaError_t Launch<G>::face_vis(const MortarC *mc, int nm, double *VF, const double *nrm, cudaStream_t s) {
  if (nm <= 0) return cudaSuccess;
  const long long n = (long long)nm * G * G;
  k_face_vis<G><<<(unsigned)((n + 127) / 128), 128, 0, s>>>(mc, nm, VF, nrm);
  return cudaGetLastError();
}

template <int G>
cudaError_t Launch<G>::face_inv_cut(const MortarCut *mc, int nm, double *QF, double *FF, const double *ghost,
                                    const double *nh, const double *nrm, double gamma, cudaStream_t s) {
  if (nm <= 0) return cudaSuccess;
  const long long n = (long long)nm * G * G;
  k_face_inv_cut<G><<<(unsigned)((n + 127) / 128), 128, 0, s>>>(mc, nm, QF, FF, ghost, nh, nrm, gamma);
  return cudaGetLastError();
}

template <int G>
cudaError_t Launch<G>::face_vis_cut(const MortarCut *mc, int nm, double *VF, const double *ghost, const double *nrm,
                                    cudaStream_t s) {
  if (nm <= 0) return cudaSuccess;
  const long long n = (long long)nm * G * G;
  k_face_vis_cut<G><<<(unsigned)((n + 127) / 128), 128, 0, s>>>(mc, nm, VF, ghost, nrm);
  return cudaGetLastError();
}

template <int G>
cudaError_t Launch<G>::face_bnd_inv(const MortarB *mb, int nm, double *QF, double *FF, const double *nh,
                                    const double *nrm, const double *qext, const BndPhys &P, cudaStream_t s) {
  if (nm <= 0) return cudaSuccess;
  const long long n = (long long)nm * G * G;
  k_face_bnd_inv<G><<<(unsigned)((n + 127) / 128), 128, 0, s>>>(mb, nm, QF, FF, nh, nrm, qext, P);
  return cudaGetLastError();
}

template <int G>
cudaError_t Launch<G>::face_bnd_vis(const MortarB *mb, int nm, double *VF, const double *nrm, const double *fvext,
                                    cudaStream_t s) {
  if (nm <= 0) return cudaSuccess;
  const long long n = (long long)nm * G * G;
  k_face_bnd_vis<G><<<(unsigned)((n + 127) / 128), 128, 0, s>>>(mb, nm, VF, nrm, fvext);
  return cudaGetLastError();
}

}  // namespace dsem

#define DSEM_INSTANTIATE(GG) template struct dsem::Launch<GG>;
