// pp_fused.cuh -- tiled fused forward + adjoint step (included by pp_tiled_fused.cu).
//
// loss = sum_{b,c,v} (pull(f_c, phi)[v] - g_c[v])^2, df = push(2 r), and
// dphi[v] = sum_c 2 r_c grad pull(f_c)[v]: the forward pull, the pull rrule's
// two cotangents (src/pushpull_pb.jl:11-18) and the loss of the differentiable
// step, in one pass over phi, f and g.
//
// A CTA takes a tile: the deformation and the target stream in like the push
// kernels' (pp_push.cuh); the image box is loaded row by row into shared memory
// and serves the value and the gradient of every voxel; the residuals replace the
// targets in the tile's ring words and are then scattered through push_channel,
// two fixed-point words per element, into an accumulator with the box's pitches.
// Taking the scatter after all residuals of the tile are known lets their actual
// size set the scale: the pass over the image for max|f| that a scale in advance
// needs is gone.  Four CTAs of 128 threads per SM cover each other's phases (the
// registers of six made the quadratic kernel spill, and three words per element leave
// room for four).  160x192x160, GB300, with that pass and 256-thread CTAs / here:
// quadratic 282 / 240 us, cubic 483 / 382; quartic 128^3 409 / 295.
#pragma once

#include "pp_push.cuh"

namespace pp {
namespace {

// Per-voxel global-memory version of one channel (tiles whose box does not fit):
// returns the residual r and the gradient; scatters 2 r into df with atomics.
// Inlined, with the rolled contraction and a rolled z loop in the scatter, so
// that the fallback costs the tiled kernel no registers.
template <int DP, typename IT>
__device__ __forceinline__ float fused_voxel_global(const LaunchArgs& a, int b, int c, long long v, float x0,
                                                    float x1, float x2, float gv, float (&grad)[3]) {
    const Geometry& g = a.g;
    const IT sy = (IT)g.d0[0];
    const IT sz = (IT)(g.d0[0] * g.d0[1]);
    int b0, b1, b2;
    bnd_code(a, c, b0, b1, b2);
    Axis<DP, 1, IT> ax, ay, az;
    ax.setup(x0, g.dp[0], b0, g.d0[0], (IT)1);
    ay.setup(x1, g.dp[1], b1, g.d0[1], sy);
    az.setup(x2, g.dp[2], b2, g.d0[2], sz);
    const float* f0 = a.in + ((long long)b * g.nc + c) * g.n0;
    IT zo[DP];
#pragma unroll
    for (int i = 0; i < DP; ++i) zo[i] = az.off[i];
    float r[6];
    contract_rolled<kPullValGrad, DP, 1>(
        ax, ay, az,
        [&](int j, float (&f)[DP]) {
#pragma unroll
            for (int i = 0; i < DP; ++i) f[i] = __ldg(f0 + (zo[0] + ay.off[j] + ax.off[i]));
        },
        [&]() {
#pragma unroll
            for (int i = 0; i + 1 < DP; ++i) zo[i] = zo[i + 1];
        },
        r);
    grad[0] = r[0];
    grad[1] = r[1];
    grad[2] = r[2];
    const float res = r[3] - gv;
    const float d = 2.f * res;
    if (finitef(d)) {
        float* df = a.out + ((long long)b * g.nc + c) * g.n0;
#pragma unroll 1
        for (int k = 0; k < DP; ++k) {
#pragma unroll
            for (int j = 0; j < DP; ++j) {
                const float cb = d * (ay.w[j] * az.w[0]);
#pragma unroll
                for (int i = 0; i < DP; ++i) atomicAdd(df + (az.off[0] + ay.off[j] + ax.off[i]), cb * ax.w[i]);
            }
#pragma unroll
            for (int i = 0; i + 1 < DP; ++i) {
                az.w[i] = az.w[i + 1];
                az.off[i] = az.off[i + 1];
            }
        }
    }
    return res;
}

constexpr int kFusedCtas = 4;

template <int DP, typename IT, bool TMA>
__global__ void __launch_bounds__(kPushThreads, kFusedCtas) k_fused_tiled(const __grid_constant__ LaunchArgs a,
                                                                             const __grid_constant__ TileGrid t,
                                                                             const __grid_constant__ CUtensorMap phimap,
                                                                             const __grid_constant__ CUtensorMap gmap) {
    extern __shared__ __align__(128) float4 smem4[];
    constexpr int NW = kPushThreads / 32;
    __shared__ int wrec[NW][8];
    __shared__ double dred[NW];
    __shared__ __align__(8) unsigned long long bars8[4];
    __shared__ int s_abort;
    const Geometry& g = a.g;
    const long long n1 = g.n1;
    const int G = gridDim.x, T0 = blockIdx.x, nv = t.nv;
    const int ntl = T0 < t.ntiles ? (t.ntiles - T0 + G - 1) / G : 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double loss = 0.0;

    float* ring = reinterpret_cast<float*>(smem4);
    const int slot_floats = 4 * nv;                  // deformation + channel-0 target
    float* img = ring + t.stages * slot_floats;      // image box
    float* accf = img + t.cap;                       // adjoint accumulator
    const unsigned bars = smem_addr(bars8);
    for (int i = threadIdx.x; i < (t.cap >> 1); i += kPushThreads)
        reinterpret_cast<float4*>(accf)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (threadIdx.x == 0) {
        s_abort = 0;
        if (TMA) {
            for (int k = 0; k < t.stages; ++k) mbar_init(bars + 8u * k, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    __syncthreads();
    for (int j = 0; j < t.stages; ++j)
        push_ring_fill<1, TMA, IT, false>(ring, slot_floats, t.stages, bars, j, T0 + j * G, j < ntl, a, a.up, t, phimap,
                                          gmap);

    for (int j = 0; j < ntl; ++j) {
        const TileOrigin o = tile_origin(t, T0 + j * G);
        float* slot = ring + (j % t.stages) * slot_floats;
        float* vslot = slot + 3 * nv;
        if constexpr (TMA) {
            if (!mbar_wait(bars + 8u * (j % t.stages), (unsigned)((j / t.stages) & 1))) s_abort = 1;
        } else {
            wait_groups(t.stages - 1);
        }
        const PushTile pt(o, t, g);
        const PushPos<false> pos{slot, nv, nullptr};

        // ---- footprint box ---------------------------------------------------
        int mn[3], mx[3];
        float ssum = 0.f, smax = 0.f;
        {
            const float inf = __int_as_float(0x7f800000);
            float lo[3] = {inf, inf, inf}, hi[3] = {-inf, -inf, -inf};
#pragma unroll 4
            for (int lin = threadIdx.x; lin < nv; lin += kPushThreads) {
                float x[3];
                const bool ok = pos(g, pt, lin, x[0], x[1], x[2]) & pt.inside(lin);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    lo[k] = fminf(lo[k], ok ? x[k] : inf);
                    hi[k] = fmaxf(hi[k], ok ? x[k] : -inf);
                }
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                mn[k] = float_key(lo[k]);
                mx[k] = float_key(hi[k]);
            }
        }
        tile_combine(wrec, true, mn, mx, ssum, smax);
        if (s_abort) break;
        PushBox box;
        if (box_place<DP>(mn, mx, g, box)) box_pitches(t, t.cap, g, box);
        float* dp = a.out2 + (long long)o.b * 3 * n1;
        for (int c = 0; c < g.nc; ++c) {
            int b0, b1, b2;
            bnd_code(a, c, b0, b1, b2);
            const float* f0 = a.in + ((long long)o.b * g.nc + c) * g.n0;
            const float* gc = a.up + ((long long)o.b * g.nc + c) * n1;
            if (c > 0) __syncthreads();   // channel c - 1 is done with the box and the accumulator
            RowBox rb{{box.lo[0], box.lo[1], box.lo[2]}, {box.e[0], box.e[1], box.e[2]}, box.P, box.Q, 0, false};
            if (box.mode == 1) {
                rb.base = box_base(box, g, f0);
                rb.fold = !(box.yin && box.zin);
                load_rows<kPushThreads, IT>(rb, g, b0, b1, b2, f0, img, threadIdx.x);
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncthreads();
                if ((b0 == 2 && !box.xin) || (b1 == 2 && !box.yin) || (b2 == 2 && !box.zin)) {
                    sign_rows<kPushThreads>(rb, g, b0, b1, b2, img, threadIdx.x);
                    __syncthreads();
                }
            }
            // ---- values, residuals and the deformation's cotangent -------------
            ssum = smax = 0.f;
            const unsigned ibase = smem_addr(img) + 4u * rb.base;
#pragma unroll 1
            for (int lin = threadIdx.x; lin < nv; lin += kPushThreads) {
                if (!pt.inside(lin)) continue;
                const IT v = pt.index<IT>(lin);
                float x0, x1, x2;
                if (!pos(g, pt, lin, x0, x1, x2)) {
                    loss += (double)qnan();   // pull is NaN here, and so is the loss
                    if (c == 0) dp[v] = dp[v + n1] = dp[v + 2 * n1] = qnan();
                    continue;
                }
                const float gv = c == 0 ? vslot[lin] : __ldg(gc + v);
                float res, grad[3];
                if (box.mode == 1) {
                    W3<DP, 1> wx, wy, wz;
                    const int ox = spline_taps32<DP, 1>(x0, wx.w, wx.dw, wx.hw) - box.lo[0];
                    const int oy = spline_taps32<DP, 1>(x1, wy.w, wy.dw, wy.hw) - box.lo[1];
                    const int oz = spline_taps32<DP, 1>(x2, wz.w, wz.dw, wz.hw) - box.lo[2];
                    float r[6];
                    contract_smem<kPullValGrad, DP>(wx, wy, wz, ibase + 4u * (unsigned)(oz * box.Q + oy * box.P + ox),
                                                    4u * box.P, 4u * box.Q, r);
                    res = r[3] - gv;
                    grad[0] = r[0];
                    grad[1] = r[1];
                    grad[2] = r[2];
                } else {
                    res = fused_voxel_global<DP, IT>(a, o.b, c, (long long)v, x0, x1, x2, gv, grad);
                }
                loss += (double)(res * res);
                const float d = 2.f * res;
                vslot[lin] = d;
                const float s1 = finitef(d) ? fabsf(d) : 0.f;
                ssum += s1;
                smax = fmaxf(smax, s1);
                float q[3] = {0.f, 0.f, 0.f};
                if (c > 0) {   // the same thread wrote the earlier channels' sum
                    q[0] = dp[v];
                    q[1] = dp[v + n1];
                    q[2] = dp[v + 2 * n1];
                }
                dp[v] = fmaf(d, grad[0], q[0]);
                dp[v + n1] = fmaf(d, grad[1], q[1]);
                dp[v + 2 * n1] = fmaf(d, grad[2], q[2]);
            }
            if (box.mode == 1) {
                tile_combine(wrec, false, mn, mx, ssum, smax);
                push_channel<DP, kPush, IT>(g, t, pt, pos, vslot, box, b0, b1, b2,
                                            a.out + ((long long)o.b * g.nc + c) * g.n0, accf, ssum, smax);
            }
        }
        if (TMA) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // residuals, then the next copy
        __syncthreads();   // ring slot j, the box and the accumulator are free
        push_ring_fill<1, TMA, IT, false>(ring, slot_floats, t.stages, bars, j + t.stages, T0 + (j + t.stages) * G,
                                          j + t.stages < ntl, a, a.up, t, phimap, gmap);
    }
    if constexpr (!TMA) asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    // this CTA's loss partial
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, off);
    if (lane == 0) dred[warp] = loss;
    __syncthreads();
    if (threadIdx.x == 0) {
        double sum = 0.0;
        for (int w = 0; w < NW; ++w) sum += dred[w];
        a.partial[blockIdx.x] = sum;
    }
}

// Tile grid, shared memory and CTAs of a fused launch.
TileGrid fused_grid(const LaunchArgs& a, TileCfg c, size_t& smem, int& ctas) {
    if (c.automatic) c = fused_own_tile(a);
    // a budget set by the caller: three words per element and one ring slot in 227 KB
    const int room = (int)((225 * 1024 - ((size_t)16 << (c.lx + c.ly + c.lz))) / 12) & ~3;
    if (c.cap > room) c.cap = room;
    TileGrid t = make_grid(a, c);
    t.pmod = (1 << c.lx) & 31;
    const int most = kFusedCtas;
    const size_t slot = (size_t)4 * t.nv * 4, boxes = (size_t)3 * c.cap * 4;
    t.stages = 4;
    while (t.stages > 1 && t.stages * slot + boxes > (226 / most - 1) * 1024) --t.stages;
    smem = t.stages * slot + boxes;
    long long per_sm = (228LL * 1024) / (long long)(smem + 1536);
    per_sm = per_sm < 1 ? 1 : (per_sm > most ? most : per_sm);
    const long long want = per_sm * sm_count();
    ctas = (int)(t.ntiles < want ? t.ntiles : want);
    return t;
}

template <int DP, typename IT>
cudaError_t launch_fused_dp(const LaunchArgs& a, const TileCfg& c, cudaStream_t s, int grid) {
    CUtensorMap phimap, gmap;
    std::memset(&phimap, 0, sizeof phimap);
    std::memset(&gmap, 0, sizeof gmap);
    size_t smem;
    int ctas;
    const TileGrid t = fused_grid(a, c, smem, ctas);
    const bool tma = encode_tile_map(&phimap, a.phi, a.g.d1, 3LL * a.g.nb, t, 3) &&
                     encode_tile_map(&gmap, a.up, a.g.d1, (long long)a.g.nc * a.g.nb, t, 1);
    cudaError_t e;
    if (tma) {
        auto k = k_fused_tiled<DP, IT, true>;
        if ((e = opt_in(k, smem)) != cudaSuccess) return e;
        k<<<grid, kPushThreads, smem, s>>>(a, t, phimap, gmap);
    } else {
        auto k = k_fused_tiled<DP, IT, false>;
        if ((e = opt_in(k, smem)) != cudaSuccess) return e;
        k<<<grid, kPushThreads, smem, s>>>(a, t, phimap, gmap);
    }
    return cudaGetLastError();
}

}  // namespace
}  // namespace pp
