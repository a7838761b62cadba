// pp_direct.cu -- pull / pull_grad / pull_hess / push / push_grad, per sample voxel
// against global memory.
//
// The general path: any degree triple (including anisotropic ones), any sample
// grid shape (the host-pointer ABI passes only n1), any deformation.  Weights are
// derived once per voxel and reused for every channel (the reference relaunches
// per channel and recomputes them, ext/pushpull_gpu.jl:37-49); boundary signs are
// folded into the weights so each tap is one load (or one reduction) and one FMA.
//
// Reference kernels replaced: pull_element, pullg_element, pullh_element,
// push_element, pushg_element (artifacts/C/pushpull.cu:33-163).
#include "pp_voxel.cuh"

namespace pp {
namespace {

// Is a launch that runs only where the sampled boxes overflow (a.sample) to run?  All
// threads of the block.
template <int DP, int OP>
__device__ __forceinline__ bool sampled_in(const LaunchArgs& a) {
    __shared__ int s_run;
    if (threadIdx.x < 32) {
        const bool over = sampled_overflow<DP, OP>(a);
        if (threadIdx.x == 0) s_run = over;
    }
    __syncthreads();
    return s_run;
}

template <int DP, int OP, typename IT>
__global__ void __launch_bounds__(256, DP >= 4 ? 2 : 0) k_pull_direct(LaunchArgs a) {
    if (DP > 0 && a.sample && !sampled_in<DP, OP>(a)) return;
    const Geometry& g = a.g;
    const long long n1 = g.n1;
    const int b = blockIdx.y;
    const float* phi = a.phi + (long long)b * 3 * n1;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < n1;
         v += (long long)gridDim.x * blockDim.x) {
        float x0, x1, x2;
        if (!load_valid(__ldg(phi + v), __ldg(phi + v + n1), __ldg(phi + v + 2 * n1), g, x0, x1, x2))
            pull_voxel_nan<OP>(a, b, v);
        else
            pull_voxel_global<DP, OP, IT>(a, b, v, x0, x1, x2);
    }
}

// A voxel whose taps do not all lie inside the image: the general per-voxel path,
// out of line so that its 64-bit folding does not weigh on the registers of the
// common one.
template <int DP, int OP>
__device__ __noinline__ void pull_voxel_folded(const LaunchArgs& a, int b, long long v, float x0, float x1, float x2) {
    pull_voxel_global<DP, OP, int>(a, b, v, x0, x1, x2);
}

// Weights of one voxel whose taps all lie inside the image.
template <int DP, int ORD>
struct InWeights {
    float w[DP];
    float dw[ORD >= 1 ? DP : 1];
    float hw[ORD >= 2 ? DP : 1];
};

// The pull family at one to three taps per axis for images of fewer than 2^31
// elements.  V voxels per thread, one block width apart, so that every load of a warp is
// contiguous at any alignment while a thread keeps 12 V bytes of deformation
// reads in flight.  Voxels whose taps all lie inside the image take a path of
// 32-bit offsets from one address with weights shared by the channels; the others
// the general one.  The arithmetic is pull_voxel_global's, bit for bit.
// What bounds it is latency (a DRAM load, then dependent L2 gathers) and, from two
// taps on, the gathers' L1 wavefronts.  GB300, 181x217x181, one channel, pull /
// pull_grad, us, against one voxel per thread with folded 64-bit indices: degree 0
// 76 / 81 -> 38 / 50 (192^3: 42 / 52 with 16-byte loads of four consecutive voxels
// per thread, which odd sizes cannot use, 38 / 50 here), degree 1 91 / 140 -> 72 /
// 107, degree 2 189 / 234 -> 124 / 154.  At four and five taps the 64 or 125
// gathers in flight leave no registers for it (cubic 128^3 97 us, k_pull_direct 72).
template <int DP, int OP_, int V>
__global__ void __launch_bounds__(256, DP == 3 && op_order(OP_) <= 1 && !pull_is_dot<OP_>() ? 3 : 0) k_pull_lean(const __grid_constant__ LaunchArgs a) {
    constexpr int OP = pull_base_op<OP_>();
    constexpr int ORD = op_order(OP);
    if (a.sample && !sampled_in<DP, OP_>(a)) return;
    const Geometry& g = a.g;
    const long long n1 = g.n1;
    const int b = blockIdx.y;
    const int dx = (int)g.d0[0] - DP, dy = (int)g.d0[1] - DP, dz = (int)g.d0[2] - DP;
    const int sy = (int)g.d0[0], sz = (int)(g.d0[0] * g.d0[1]);
    const float* phi = a.phi + (long long)b * 3 * n1;
    const float* fb = a.in + (long long)b * g.nc * g.n0;
    for (long long v0 = (long long)blockIdx.x * (256 * V) + threadIdx.x; v0 < n1; v0 += (long long)gridDim.x * (256 * V)) {
        float X[V][3];
#pragma unroll
        for (int u = 0; u < V; ++u) {
            const long long v = v0 + u * 256;
            const bool in = V == 1 || v < n1;
#pragma unroll
            for (int k = 0; k < 3; ++k) X[u][k] = in ? __ldg(phi + v + k * n1) : qnan();
        }
        int at[V];   // element of the first tap; -1 nothing left to do
        InWeights<DP, ORD> wx[V], wy[V], wz[V];
#pragma unroll
        for (int u = 0; u < V; ++u) {
            const long long v = v0 + u * 256;
            float x0, x1, x2;
            const bool ok = load_valid(X[u][0], X[u][1], X[u][2], g, x0, x1, x2);
            const int ox = spline_taps32<DP, ORD>(x0, wx[u].w, wx[u].dw, wx[u].hw);
            const int oy = spline_taps32<DP, ORD>(x1, wy[u].w, wy[u].dw, wy[u].hw);
            const int oz = spline_taps32<DP, ORD>(x2, wz[u].w, wz[u].dw, wz[u].hw);
            const bool inside = ok & (ox >= 0) & (oy >= 0) & (oz >= 0) & (ox <= dx) & (oy <= dy) & (oz <= dz);
            at[u] = inside ? oz * sz + oy * sy + ox : -1;
            if (!inside && (V == 1 || v < n1)) {
                if (ok) pull_voxel_folded<DP, OP_>(a, b, v, x0, x1, x2);
                else pull_voxel_nan<OP_>(a, b, v);
            }
        }
        float acc[pull_is_dot<OP_>() ? V : 1][3];
        if constexpr (pull_is_dot<OP_>()) {
#pragma unroll
            for (int u = 0; u < V; ++u) acc[u][0] = acc[u][1] = acc[u][2] = 0.f;
        }
#pragma unroll 1
        for (int c = 0; c < g.nc; ++c) {
            const float* f0 = fb + (long long)c * g.n0;
#pragma unroll
            for (int u = 0; u < V; ++u) {
                if (at[u] < 0) continue;
                const float* p = f0 + at[u];
                float r[6];
                contract_rolled<OP, DP, DP>(
                    wx[u], wy[u], wz[u],
                    [&](int j, float(&f)[DP]) {
#pragma unroll
                        for (int i = 0; i < DP; ++i) f[i] = __ldg(p + j * sy + i);
                    },
                    [&]() { p += sz; }, r);
                if constexpr (pull_is_dot<OP_>()) dot_accumulate<OP_>(a, b, c, v0 + u * 256, r, acc[u]);
                else pull_store<OP>(pull_out<OP_>(a, b, c, v0 + u * 256), n1, r);
            }
        }
        if constexpr (pull_is_dot<OP_>()) {
#pragma unroll
            for (int u = 0; u < V; ++u) {
                if (at[u] < 0) continue;
                float* o = pull_out<OP_>(a, b, 0, v0 + u * 256);
                o[0] = acc[u][0];
                o[n1] = acc[u][1];
                o[2 * n1] = acc[u][2];
            }
        }
    }
}

template <int DP, int OP, typename IT>
__global__ void __launch_bounds__(256) k_push_direct(LaunchArgs a) {
    const Geometry& g = a.g;
    const long long n1 = g.n1;
    const int b = blockIdx.y;
    const float* phi = a.phi + (long long)b * 3 * n1;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < n1;
         v += (long long)gridDim.x * blockDim.x) {
        float x0, x1, x2;
        if (load_valid(__ldg(phi + v), __ldg(phi + v + n1), __ldg(phi + v + 2 * n1), g, x0, x1, x2))
            push_voxel_global<DP, OP, IT>(a, b, v, x0, x1, x2);
    }
}

template <int DP, int OP, typename IT, bool PUSH>
void launch_one(const LaunchArgs& a, dim3 grid, cudaStream_t s) {
    if constexpr (PUSH) {
        k_push_direct<DP, OP, IT><<<grid, 256, 0, s>>>(a);
    } else if constexpr (DP > 0 && DP <= 3 && sizeof(IT) == 4) {
        // Small volumes: a warp of 32 voxels along x nearly always holds some at the
        // border and takes both of k_pull_lean's paths, so that folding every voxel is
        // faster (64^3, k_pull_lean / here, us: linear pull 8.4 / 6.5, three channels
        // 12.4 / 10.4, quadratic pull_hess 16.5 / 12.6; from 80^3 on within a tenth, and
        // a block that stays inside a larger image gains by k_pull_lean: 96^3 out of 192^3
        // quadratic pull 14.5 / 22.8).  Four voxels per thread only at one tap per axis
        // and only when that still fills the chip (degree 0, one / four: 121^3 19 / 17,
        // 181x217x181 66 / 38, 64^3 9 / 11; 64^3 here 6).
        if (a.g.n1 * a.g.nb < (DP == 1 ? 1LL << 20 : 3LL << 17)) {
            k_pull_direct<DP, OP, IT><<<grid, 256, 0, s>>>(a);
        } else if constexpr (DP == 1) {
            const long long blocks = (a.g.n1 + 1023) / 1024, cap = (long long)sm_count() * 8;
            k_pull_lean<DP, OP, 4><<<dim3((unsigned)(blocks < cap ? blocks : cap), grid.y), 256, 0, s>>>(a);
        } else {
            k_pull_lean<DP, OP, 1><<<grid, 256, 0, s>>>(a);
        }
    } else {
        k_pull_direct<DP, OP, IT><<<grid, 256, 0, s>>>(a);
    }
}

template <int OP, typename IT, bool PUSH>
cudaError_t dispatch_dp(const LaunchArgs& a, dim3 grid, cudaStream_t s) {
    const int d = a.g.dp[0];
    const bool iso = a.g.dp[1] == d && a.g.dp[2] == d;
    switch (iso ? d : 0) {
        case 1: launch_one<1, OP, IT, PUSH>(a, grid, s); break;
        case 2: launch_one<2, OP, IT, PUSH>(a, grid, s); break;
        case 3: launch_one<3, OP, IT, PUSH>(a, grid, s); break;
        case 4: launch_one<4, OP, IT, PUSH>(a, grid, s); break;
        case 5: launch_one<5, OP, IT, PUSH>(a, grid, s); break;
        default: launch_one<0, OP, IT, PUSH>(a, grid, s); break;
    }
    return cudaGetLastError();
}

dim3 direct_grid(int op, const LaunchArgs& a) {
    const long long blocks_needed = (a.g.n1 + 255) / 256;
    long long cap = (long long)sm_count() * 8;
    // only where the sample says so: no more blocks than fit at once, which look at it
    // once each (eight per SM take three rounds: 6 us more)
    if (a.sample) cap = ((long long)sm_count() * (a.g.dp[0] > 3 ? 2 : (op <= kPullGrad ? 3 : 6)) + a.g.nb - 1) / a.g.nb;
    return dim3((unsigned)(blocks_needed < cap ? blocks_needed : cap), (unsigned)a.g.nb);
}

}  // namespace

cudaError_t launch_pull_direct(int op, const LaunchArgs& a, cudaStream_t s) {
    const dim3 grid = direct_grid(op, a);
    const bool small = a.g.n0 < (1LL << 31) - 1;
    switch (op) {
        case kPull: return small ? dispatch_dp<kPull, int, false>(a, grid, s)
                                 : dispatch_dp<kPull, long long, false>(a, grid, s);
        case kPullGrad: return small ? dispatch_dp<kPullGrad, int, false>(a, grid, s)
                                     : dispatch_dp<kPullGrad, long long, false>(a, grid, s);
        case kPullHess: return small ? dispatch_dp<kPullHess, int, false>(a, grid, s)
                                     : dispatch_dp<kPullHess, long long, false>(a, grid, s);
        case kPullGradDot: return small ? dispatch_dp<kPullGradDot, int, false>(a, grid, s)
                                        : dispatch_dp<kPullGradDot, long long, false>(a, grid, s);
        default: return small ? dispatch_dp<kPullHessDot, int, false>(a, grid, s)
                              : dispatch_dp<kPullHessDot, long long, false>(a, grid, s);
    }
}

cudaError_t launch_push_direct(int op, const LaunchArgs& a, cudaStream_t s) {
    const dim3 grid = direct_grid(op, a);
    const bool small = a.g.n0 < (1LL << 31) - 1;
    if (op == kPush)
        return small ? dispatch_dp<kPush, int, true>(a, grid, s) : dispatch_dp<kPush, long long, true>(a, grid, s);
    return small ? dispatch_dp<kPushGrad, int, true>(a, grid, s) : dispatch_dp<kPushGrad, long long, true>(a, grid, s);
}

}  // namespace pp
