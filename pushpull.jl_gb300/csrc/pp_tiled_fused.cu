// pp_tiled_fused.cu -- tiled fused forward + adjoint step kernels
// (pp_fused.cuh).
#include "pp_fused.cuh"

namespace pp {

// The tile and budget (floats of the image box, words of the accumulator) measured
// best: 160x192x160 quadratic, us: 16x8x4 229, 8x8x8 241, 16x4x8 237, 8x16x4 250,
// 32x4x4 248; with five CTAs per SM and a larger budget 237, with four 231.
TileCfg fused_own_tile(const LaunchArgs& a) { return TileCfg{4, 3, 2, a.g.dp[0] <= 3 ? 3072 : 4864}; }

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
