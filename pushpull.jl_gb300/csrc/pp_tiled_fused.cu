// pp_tiled_fused.cu -- tiled fused forward + adjoint step kernels
// (pp_fused.cuh).
#include "pp_fused.cuh"

namespace pp {

// The tile and budget (floats of the image box; the accumulator has two words for each)
// measured best.  160x192x160, us, with the best budget of each shape: quadratic 16x8x4
// 240, 8x8x8 241, 16x4x8 244; cubic 382, 385, 390; quartic 128^3 8x8x8 295, 8x16x4 321,
// 16x8x4 326.
TileCfg fused_own_tile(const LaunchArgs& a) {
    const int dp = a.g.dp[0];
    return dp == 5 ? TileCfg{3, 3, 3, 4864} : TileCfg{4, 3, 2, dp <= 3 ? 3328 : 3840};
}

int fused_tiled_grid(const LaunchArgs& a, const TileCfg& c) {
    size_t smem;
    int ctas;
    (void)fused_grid(a, c, smem, ctas);
    return ctas;
}

cudaError_t launch_fused_tiled(const LaunchArgs& a, const TileCfg& t, cudaStream_t s, int grid) {
    const bool small = a.g.n0 < (1LL << 31) - 1 && a.g.n1 < (1LL << 31) - 1;
    switch (a.g.dp[0]) {
        case 1: return small ? launch_fused_dp<1, int>(a, t, s, grid) : launch_fused_dp<1, long long>(a, t, s, grid);
        case 2: return small ? launch_fused_dp<2, int>(a, t, s, grid) : launch_fused_dp<2, long long>(a, t, s, grid);
        case 3: return small ? launch_fused_dp<3, int>(a, t, s, grid) : launch_fused_dp<3, long long>(a, t, s, grid);
        case 4: return small ? launch_fused_dp<4, int>(a, t, s, grid) : launch_fused_dp<4, long long>(a, t, s, grid);
        default: return small ? launch_fused_dp<5, int>(a, t, s, grid) : launch_fused_dp<5, long long>(a, t, s, grid);
    }
}

unsigned status_fused(bool reset) { return unit_status(reset); }

}  // namespace pp
