// dsem_shapes.h -- which volume kernel a launch runs and with how many warps per element.
// Host-side rules only (no CUDA): the launchers switch on them, and a CPU test reads them.
#pragma once

namespace dsem {

constexpr int SM_COUNT = 148;  // multiprocessors of a B200

// launch shapes of the diagonal volume kernel the autotuner chooses from (0 the default)
constexpr int VOL_VARIANTS = 5;

// Launch shapes of k_vol_mma (0..5) and k_vol_mma_gen (6, 7): warps per element and the elements
// an SM must hold at once, which sets the register budget.
// 0..4: dsem_autotune times 1..4 against the default 0 for p = 4, 6, 8.  Shared memory allows 2
// elements per SM at p >= 7, 4 at p = 6, 6 at p = 5 and 10 at p = 4.  Measured, ms of shapes 0..4
// (22^3 of p = 8, 24^3 of p = 6, 32^3 of p = 4): 1.127 1.156 1.180 1.233 1.307; 0.745 0.762 0.946
// 0.739 0.854; 0.640 0.708 0.644 0.700 0.671.  Every shape evaluates each value with the same chain.
// MMA_WIDE: variant 0 for launches of at most SM_COUNT * mma_minb elements, which do not
// fill the GPU: more warps work on one element, and its latency is the launch's.  Measured against
// variant 1's or 0's shape, us: 4^3 elements of p = 8 23.8 (8 warps: 27), p = 6 15.6 (3 warps:
// 24.7), p = 4 10.4 (2 warps: 16.5); p = 4 at 512 elements, which shape 3 still holds at
// once, 16.5 with it (2 warps: 19.6); a step of 343 elements with a viscosity model 121.2 us
// against 147.9 (Smagorinsky), 125.2 against 153.8 (entropy viscosity).
// MMA_GEN, MMA_GEN_WIDE: k_vol_mma_gen (20 shared fields), the latter for the same reason.
constexpr int MMA_WIDE = 5, MMA_GEN = 6, MMA_GEN_WIDE = 7;
constexpr int mma_warps(int G, int V) {
  return V == MMA_GEN        ? (G >= 8 ? 12 : (G == 7 ? 4 : 2))
         : V == MMA_GEN_WIDE ? (G >= 7 ? 12 : 4)
         : G >= 8 ? (V == MMA_WIDE ? 16 : (V == 0 ? 8 : (V == 1 ? 6 : (V == 2 ? 7 : (V == 3 ? 5 : 4)))))
         : G >= 6 ? (V == MMA_WIDE ? (G == 7 ? 12 : 8) : (V == 0 ? 4 : (V == 1 ? 3 : (V == 2 ? 2 : (V == 3 ? 5 : 6)))))
         : G == 5 ? (V == MMA_WIDE ? 8 : (V <= 2 ? 2 : (V == 3 ? 4 : 3)))
                  : (V == MMA_WIDE ? 4 : 2);
}
constexpr int mma_minb(int G, int V) {
  return V == MMA_GEN        ? (G >= 8 ? 1 : (G == 7 ? 3 : (G == 6 ? 6 : 8)))
         : V == MMA_GEN_WIDE ? (G >= 7 ? 1 : 3)
         : G >= 8 ? (V == MMA_WIDE ? 1 : 2)
         : G >= 6 ? (V == MMA_WIDE ? (G == 7 ? 1 : 2) : (V == 3 ? 3 : (V == 4 ? 2 : 4)))
         : G == 5 ? (V == MMA_WIDE ? 2 : (V == 0 ? 8 : (V == 1 ? 6 : (V == 2 ? 10 : (V == 3 ? 4 : 5)))))
                  : (V == MMA_WIDE ? 4 : 8);
}

// Full metrics at p = 4 and 5 up to here: k_vol, 256 threads per element.  Its thread-per-point
// phases have the shorter chain when an SM holds one element (p = 5 also when it takes two in
// turn): a tile of p = 5 costs what one of p = 6 does (five interior points in eight columns).
// Measured, us per volume launch, k_vol against the best of ten warp counts and budgets of
// k_vol_mma_gen: p = 5 at 27, 108, 147 elements 16.7, 17.5, 18.1 against 20.5; at 150, 216, 294
// 26.8, 28.6, 29.0 against 26.4, 27.5, 27.4 with 6 warps and 28.7, 29.0, 29.0 with the wide shape;
// at 343 39.2 against 35.5 (wide).  p = 4 at 27, 108, 147 elements 14.4, 14.8, 15.5 against 14.5,
// 15.1, 15.9, and 15.8, 16.5, 17.9 with the wide shape; at 150 23.4 against 18.6 (wide).
constexpr int vol_point_max(int G) { return G == 5 ? SM_COUNT : (G == 6 ? 2 * SM_COUNT : 0); }

// orders whose diagonal kernel has the shapes 1..4 (p = 4, 6, 8)
constexpr bool vol_has_variants(int G) { return G == 5 || G == 7 || G == 9; }

// The shape a launch of nel elements of G = p + 1 takes: one of the above, or VOL_POINT for the
// kernels with a thread per point (k_vol_diag, k_vol): p = 1, 2, whose lines are too few for the
// 8-line tiles, and small launches of full metrics at p = 4, 5.  ev: entropy viscosity (its launches have the default shapes only).
constexpr int VOL_POINT = -1;
constexpr int vol_shape(int G, bool diag, int nel, bool ev, int variant) {
  if (G < 4) return VOL_POINT;
  if (!diag) {  // (p >= 7: one shape)
    if (nel <= vol_point_max(G)) return VOL_POINT;
    return G < 8 && nel <= SM_COUNT * mma_minb(G, MMA_GEN_WIDE) ? MMA_GEN_WIDE : MMA_GEN;
  }
  if (variant > 0 && variant < VOL_VARIANTS && vol_has_variants(G) && !ev) return variant;
  if (nel <= SM_COUNT * mma_minb(G, MMA_WIDE)) return MMA_WIDE;
  if (G == 5 && nel <= SM_COUNT * mma_minb(G, 3)) return 3;  // p = 4: between the two, four warps
  return 0;
}

}  // namespace dsem
