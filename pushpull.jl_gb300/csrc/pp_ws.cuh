// pp_ws.cuh -- warp-specialised persistent pull family: pull, pull_grad,
// pull_hess, the rrule contractions pull_grad_dot / pull_hess_dot, and the
// affine pull.
//
// Included after pp_tiled_impl.cuh (whose helpers it uses) by pp_ws_pull.cu,
// pp_ws_hess.cu, pp_ws_grad_dot.cu and pp_ws_hess_dot.cu.
//
// One CTA per SM: 15 consumer warps and one producer warp (512 threads, so
// every thread keeps 128 registers).  The CTA walks tiles of 8 x 16 x 15 sample
// voxels, four per consumer thread, in (tile, channel) units:
//   * the producer warp streams each tile's deformation into a ring of
//     shared-memory slots with one TMA copy per tile (mbarrier complete_tx);
//   * every consumer warp reduces the first taps of its own voxels of tile
//     j + 1 before it evaluates tile j and publishes the warp's bounds;
//   * the producer combines the fifteen records into the tile's footprint box
//     and, for a box inside the image that fits the launch's window (24 x 24 x 26
//     for an undeformed grid, shaped to the map for an affine one),
//     stages it with one TMA copy into one of two buffers while the consumers
//     still evaluate the previous unit; it then publishes the box record;
//   * boundary boxes whose margins mirror (DCT-II, DST-II) onto elements of the
//     box itself arrive by the same TMA copy, zero-filled outside the image,
//     and the consumers complete the margins in shared memory behind
//     consumer-only named barriers;
//   * other boundary boxes (circulant margins) are loaded by the consumers when
//     they take the unit, row by row with cp.async, folded on the way, 16-byte
//     chunks where a row allows it (pitches congruent to the image's make that
//     the rule for odd extents too), then signed if a margin is DST-II;
//   * of an image whose rows are not multiples of 16 bytes, every box is loaded
//     that way, but one unit ahead: bounds are published two tiles ahead, and the
//     copies of unit q + 1 are in flight while unit q is evaluated (one producer
//     warp issuing them instead took 25 us a box);
//   * a deformation that TMA cannot address (odd x extent) is copied by the
//     consumer threads themselves, each the words of its own voxels, with
//     cp.async groups as deep as the ring.
// Interior units therefore pass no CTA-wide barrier at all.  Boxes larger than
// a buffer take the per-voxel global path for that tile.
// 181x217x181, cubic, GB300: pull 0.186 ms, pull_grad 0.217 ms (0.308 and 0.324 ms
// on the block-synchronous kernels).
//
// Reference kernels replaced: pull_element / pullg_element / pullh_element
// (artifacts/C/pushpull.cu:33-109); per-voxel math pull1 / pullg1 / pullh1
// (artifacts/C/pushpull_dev.cu:61-117); the rrule contractions replace the
// pull_grad and pull_hess temporaries of the rrules (src/pushpull_pb.jl:11-35).
#pragma once

#include <cmath>

#include "pp_tiled_impl.cuh"

namespace pp {
namespace {

constexpr int kWsCons = 480;                   // consumer threads (15 warps)
constexpr int kWsThreads = kWsCons + 32;       // plus the producer warp
constexpr int kWsV = 4;                        // sample voxels per consumer thread
// The tile is about as wide as it is deep, so that a rotated or strained footprint
// still fits the window and few samples of the last tiles are lost (192^3 cubic
// pull 156 -> 154 us, pull_grad 179 -> 175, 181x217x181 200 -> 191 against 8 x 8 x
// 30; affine pulls with rotations up to 10 degrees 191 -> 167).
// (kWsLy, kWsTy and kWsTz are shared with the per-voxel kernels: pp_kernels.cuh.)
constexpr int kWsNV = kWsCons * kWsV;          // 1920 voxels per tile
constexpr int kWsStages = 4;                   // deformation ring slots
constexpr int kWsBufs = 2;                     // box buffers
// TMA image window: row pitch kWsWinX = 24 (an undeformed 8 x 4 warp tile reads 32
// distinct banks), t.winy rows and t.winz planes, kWsRows rows at most, chosen per
// launch (ws_window); kWsCap floats per box buffer
constexpr size_t kWsSmem = (size_t)(kWsStages * 3 * kWsNV + kWsBufs * kWsCap) * sizeof(float);

__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Tile-local voxel lin (x fastest, 8 x 16 x 15) -> linear sample index, or -1.
template <typename IT>
__device__ __forceinline__ IT ws_index(const TileOrigin& o, int lin, int D0, int D1, int D2) {
    const int gx = o.x0 + (lin & 7), gy = o.y0 + ((lin >> 3) & (kWsTy - 1)), gz = o.z0 + (lin >> (3 + kWsLy));
    if (gx >= D0 || gy >= D1 || gz >= D2) return (IT)-1;
    return (IT)gx + (IT)D0 * ((IT)gy + (IT)D1 * (IT)gz);
}

// Origin of linear tile T (x fastest, batch slowest) of the tile grid.
__device__ __forceinline__ TileOrigin ws_origin(const TileGrid& t, int T) {
    const unsigned u = (unsigned)T;
    const unsigned q1 = (unsigned)(((unsigned long long)u * t.mx) >> t.sx);
    const unsigned q2 = (unsigned)(((unsigned long long)q1 * t.my) >> t.sy);
    const unsigned q3 = (unsigned)(((unsigned long long)q2 * t.mz) >> t.sz);
    TileOrigin r;
    r.x0 = (int)(u - q1 * (unsigned)t.ntx) << 3;
    r.y0 = (int)(q1 - q2 * (unsigned)t.nty) << kWsLy;
    r.z0 = (int)(q2 - q3 * (unsigned)t.ntz) * kWsTz;
    r.b = (int)q3;
    return r;
}

// Sample positions of a tile's voxels: x = phi - 1 from the tile's ring slot,
// or (AFF, the affine ops) A * (i, j, k, 1) from the voxel's grid coordinates;
// either way with the validity test.
template <bool AFF>
struct WsPos {
    const float* slot;
    const AffineMap* A;
    __device__ __forceinline__ bool operator()(const Geometry& g, const TileOrigin& o, int lin, float& x0, float& x1,
                                               float& x2) const {
        if constexpr (AFF) {
            affine_position(*A, (float)(o.x0 + (lin & 7)), (float)(o.y0 + ((lin >> 3) & (kWsTy - 1))),
                            (float)(o.z0 + (lin >> (3 + kWsLy))), x0, x1, x2);
            return position_valid(x0, x1, x2, g);
        } else {
            return load_valid(slot[lin], slot[kWsNV + lin], slot[2 * kWsNV + lin], g, x0, x1, x2);
        }
    }
};

// First-tap bounds of one consumer thread's voxels of the tile, reduced over
// its warp (every lane ends with the warp's bounds).
template <int DP, typename IT, class POS>
__device__ __forceinline__ void ws_warp_bounds(const Geometry& g, const TileOrigin& o, const POS& pos, int ctid,
                                               int D0, int D1, int D2, int (&mn)[3], int (&mx)[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        mn[k] = INT_MAX;
        mx[k] = INT_MIN;
    }
#pragma unroll
    for (int q = 0; q < kWsV; ++q) {
        const int i = ctid + q * kWsCons;
        if (ws_index<IT>(o, i, D0, D1, D2) < 0) continue;
        float x[3];
        if (!pos(g, o, i, x[0], x[1], x[2])) continue;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int f = first_tap32(x[k], DP);
            const int c = f < -kClamp ? -kClamp : (f > kClamp ? kClamp : f);
            mn[k] = min(mn[k], c);
            mx[k] = max(mx[k], c);
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        mn[k] = __reduce_min_sync(0xffffffffu, mn[k]);
        mx[k] = __reduce_max_sync(0xffffffffu, mx[k]);
    }
}

// Footprint box of a tile from the consumer warps' bound records (producer
// warp; every lane ends with the same box).
template <int DP>
__device__ __forceinline__ Box ws_tile_box(const Geometry& g, const TileGrid& t, const int (*wrec)[6], int lane) {
    constexpr int NW = kWsCons / 32;
    int mn[3], mx[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        mn[k] = __reduce_min_sync(0xffffffffu, lane < NW ? wrec[lane][k] : INT_MAX);
        mx[k] = __reduce_max_sync(0xffffffffu, lane < NW ? wrec[lane][3 + k] : INT_MIN);
    }
    Box box;
    box.S = 0.f;
    box.E = 0;
    box.tma = 0;
    box.base = 0;
    if (mn[0] > mx[0]) {   // no valid voxel in the tile
        box.mode = 0;
        box.interior = 0;
        box.xo = box.lo[0] = box.lo[1] = box.lo[2] = 0;
        box.ext[0] = box.ext[1] = box.ext[2] = 0;
        box.P = box.Q = box.size = 0;
        return box;
    }
    const int xo = mn[0] & ~3;
    const long long e0 = (long long)mx[0] + DP - xo;
    const long long e1 = (long long)mx[1] + DP - mn[1];
    const long long e2 = (long long)mx[2] + DP - mn[2];
    int interior = 0;
    if (xo >= 0 && (long long)mx[0] + DP <= g.d0[0]) interior |= 1;
    if (mn[1] >= 0 && (long long)mx[1] + DP <= g.d0[1]) interior |= 2;
    if (mn[2] >= 0 && (long long)mx[2] + DP <= g.d0[2]) interior |= 4;
    box.interior = interior;
    box.xo = xo;
    box.lo[0] = mn[0];
    box.lo[1] = mn[1];
    box.lo[2] = mn[2];
    if (t.img_tma && interior == 7 && e0 <= kWsWinX && e1 <= t.winy && e2 <= t.winz) {
        box.mode = 1;
        box.tma = 1;
        box.P = kWsWinX;
        box.Q = kWsWinX * t.winy;
        box.size = kWsCap;
        box.ext[0] = (int)e0;
        box.ext[1] = (int)e1;
        box.ext[2] = (int)e2;
        return box;
    }
    // boundary box, or an image TMA cannot address: provisional record with the
    // window's extents; the producer decides per channel how it is loaded
    const bool fits = e0 <= 4096 && e1 <= 4096 && e2 <= 4096;
    box.mode = fits ? 1 : 2;
    box.ext[0] = fits ? (int)e0 : 0;
    box.ext[1] = fits ? (int)e1 : 0;
    box.ext[2] = fits ? (int)e2 : 0;
    box.P = box.Q = box.size = 0;
    box.lo[0] = mn[0];
    return box;
}

__device__ __forceinline__ RowBox box_rows(const Box& b) {
    return RowBox{{b.xo, b.lo[1], b.lo[2]}, {b.ext[0], b.ext[1], b.ext[2]}, b.P, b.Q, b.base, (b.interior & 6) != 6};
}

// Pitches of a box that is loaded row by row (load_rows): congruent
// to the image's row and plane modulo 4 elements, so that 16-byte chunks of a row
// are aligned in both; the row pitch 8 or 24 modulo 32 (plus that remainder)
// keeps an 8 x 4 warp tile's rows in nearly disjoint banks.  Three words lie
// between rows: a row's first and last chunk may overwrite them.
__device__ __forceinline__ void ws_async_pitch(Box& box, const Geometry& g, int lo0, int e0) {
    const int rm = (int)(g.d0[0] & 3), pm = (int)((g.d0[0] * g.d0[1]) & 3);
    box.xo = lo0;
    box.ext[0] = e0;
    const int least = e0 + 3;
    int P = least + ((rm - least) & 3);
    int Pb = 8 + rm;
    while (Pb < least) Pb += 16;
    const long long e1 = box.ext[1], e2 = box.ext[2];
    long long Q = (long long)Pb * e1;
    Q += (pm - Q) & 31;
    if (Q * e2 + 8 <= kWsCap) {
        P = Pb;
    } else {
        Q = (long long)P * e1;
        Q += (pm - Q) & 3;
    }
    const bool fits = Q * e2 + 8 <= kWsCap;
    box.mode = fits ? 1 : 2;
    box.P = fits ? P : 0;
    box.Q = fits ? (int)Q : 0;
    box.size = fits ? (int)(Q * e2) : 0;
    box.tma = 3;
}

// A boundary box whose out-of-image margins all fold by a mirror (DCT-II or
// DST-II) onto elements inside the box itself can be loaded by the TMA window
// like an interior box (the margins arrive zero-filled) and completed in shared
// memory by ws_mirror_fixup.  True when the box fits the window and every
// margin qualifies; boxes with circulant margins (whose sources lie across the
// image) or margins wider than the in-image part are loaded row by row instead.
__device__ __forceinline__ bool ws_mirror_ok(const Box& box, const Geometry& g, const TileGrid& t, int b0, int b1,
                                             int b2) {
    if (box.mode != 1 || box.ext[0] > kWsWinX || box.ext[1] > t.winy || box.ext[2] > t.winz) return false;
    const int bk[3] = {b0, b1, b2};
    const int lo[3] = {box.xo, box.lo[1], box.lo[2]};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const long long d = g.d0[k], l = lo[k], e = box.ext[k];
        const long long hl = l < 0 ? -l : 0, hr = l + e > d ? l + e - d : 0;
        if (hl == 0 && hr == 0) continue;
        if (bk[k] == 0) return false;                                    // circulant
        if (hl > d || hr > d) return false;                              // more than one reflection
        if (hl > 0 && l + e < 2 * hl) return false;                      // left sources [0, hl) outside the box
        if (hr > 0 && d - hr < l) return false;                          // right sources [d - hr, d) outside
    }
    return true;
}

// Fill the margins of a TMA-loaded boundary box from their mirror images inside the box, x margins first
// (rows inside the image in y and z), then whole y-margin rows (planes inside
// in z), then whole z-margin planes, each step reading only elements the
// previous steps completed.  DST-II margins take the sign -1.  All consumer
// threads; named barrier 1 between the steps and at the end.
__device__ __forceinline__ void ws_mirror_fixup(const Box& box, const Geometry& g, int b0, int b1, int b2,
                                                float* sm, int tid, int nthreads) {
    constexpr int P = kWsWinX;
    const int Q = box.Q;
    const int e0 = box.ext[0], e1 = box.ext[1], e2 = box.ext[2];
    const int lx = box.xo, ly = box.lo[1], lz = box.lo[2];
    const int dx = (int)g.d0[0], dy = (int)g.d0[1], dz = (int)g.d0[2];
    // x margins
    const int hlx = lx < 0 ? -lx : 0, hrx = lx + e0 > dx ? lx + e0 - dx : 0, nh = hlx + hrx;
    if (nh > 0) {
        const float sx = b0 == 2 ? -1.f : 1.f;
        const int items = nh * e1 * e2;
        for (int it = tid; it < items; it += nthreads) {
            const int row = it / nh, h = it - row * nh;
            const int rz = row / e1, ry = row - rz * e1;
            const int gy = ly + ry, gz = lz + rz;
            if (gy < 0 || gy >= dy || gz < 0 || gz >= dz) continue;   // a y or z margin row: later
            const int ex = h < hlx ? h : e0 - hrx + (h - hlx);
            const int gx = lx + ex;
            const int src = (gx < 0 ? -1 - gx : 2 * dx - 1 - gx) - lx;
            float* r = sm + rz * Q + ry * P;
            r[ex] = sx * r[src];
        }
        asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
    }
    // y margin rows of the planes inside the image
    const int hly = ly < 0 ? -ly : 0, hry = ly + e1 > dy ? ly + e1 - dy : 0, nhy = hly + hry;
    if (nhy > 0) {
        const float sy = b1 == 2 ? -1.f : 1.f;
        const int items = nhy * e2 * e0;
        for (int it = tid; it < items; it += nthreads) {
            const int rowi = it / e0, x = it - rowi * e0;
            const int rz = rowi / nhy, h = rowi - rz * nhy;
            const int gz = lz + rz;
            if (gz < 0 || gz >= dz) continue;
            const int ry = h < hly ? h : e1 - hry + (h - hly);
            const int gy = ly + ry;
            const int sry = (gy < 0 ? -1 - gy : 2 * dy - 1 - gy) - ly;
            sm[rz * Q + ry * P + x] = sy * sm[rz * Q + sry * P + x];
        }
        asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
    }
    // z margin planes
    const int hlz = lz < 0 ? -lz : 0, hrz = lz + e2 > dz ? lz + e2 - dz : 0, nhz = hlz + hrz;
    if (nhz > 0) {
        const float sz = b2 == 2 ? -1.f : 1.f;
        const int per = e1 * e0;
        const int items = nhz * per;
        for (int it = tid; it < items; it += nthreads) {
            const int h = it / per, rem = it - h * per;
            const int ry = rem / e0, x = rem - ry * e0;
            const int rz = h < hlz ? h : e2 - hrz + (h - hlz);
            const int gz = lz + rz;
            const int srz = (gz < 0 ? -1 - gz : 2 * dz - 1 - gz) - lz;
            sm[rz * Q + ry * P + x] = sz * sm[srz * Q + ry * P + x];
        }
        asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
    }
}

// One consumer thread, one (tile, channel) unit of the pull family: its four
// voxels against the staged box.  The dot ops accumulate over channels in the
// output itself: channel 0 writes its term, later channels (same thread, same
// voxels) read it back and add theirs, in the order the per-voxel kernels
// accumulate in registers.
template <int DP, int OP_, typename IT, class POS>
__device__ __forceinline__ void ws_pull_unit(const LaunchArgs& a, const TileOrigin& o, int ctid, const POS& pos,
                                             int c, const Box& box, const float* sm, int D0, int D1, int D2) {
    constexpr int OP = pull_base_op<OP_>();
    constexpr int NCOMP = pull_ncomp<OP_>();
    constexpr int ORD = op_order(OP);
    const Geometry& g = a.g;
    const long long n1 = g.n1;
    const bool last = c == g.nc - 1;
    // the box record in registers: the output stores would otherwise make the
    // compiler reload it from shared memory for every voxel
    const int bmode = box.mode, bxo = box.xo, by0 = box.lo[1], bz0 = box.lo[2], bP = box.P, bQ = box.Q;
    sm += box.base;
    auto voxel = [&](int q) {
        const int lin = ctid + q * kWsCons;
        const IT v = ws_index<IT>(o, lin, D0, D1, D2);
        if (v < 0) return;
        float x0, x1, x2;
        if (!pos(g, o, lin, x0, x1, x2)) {
            if (!pull_is_dot<OP_>() || last) {
                float* out = pull_out<OP_>(a, o.b, c, (long long)v);
#pragma unroll
                for (int p = 0; p < NCOMP; ++p) out[(long long)p * n1] = qnan();
            }
            return;
        }
        if (bmode == 2) {   // box larger than a buffer: every channel from global memory, once
            if (c == 0) pull_voxel_lean<DP, OP_, IT>(a, o.b, (long long)v, x0, x1, x2);
            return;
        }
        if (bmode != 1) return;
        W3<DP, ORD> wx, wy, wz;
        const int ox = spline_taps32<DP, ORD>(x0, wx.w, wx.dw, wx.hw) - bxo;
        const int oy = spline_taps32<DP, ORD>(x1, wy.w, wy.dw, wy.hw) - by0;
        const int oz = spline_taps32<DP, ORD>(x2, wz.w, wz.dw, wz.hw) - bz0;
        const unsigned P4 = 4u * bP, Q4 = 4u * bQ;
        const unsigned p = smem_addr(sm) + 4u * (unsigned)(oz * bQ + oy * bP + ox);
        float r[6];
        contract_smem<OP, DP>(wx, wy, wz, p, P4, Q4, r);
        if constexpr (pull_is_dot<OP_>()) {
            float* out = pull_out<OP_>(a, o.b, 0, (long long)v);
            float acc[3] = {0.f, 0.f, 0.f};
            if (c > 0) {
                acc[0] = out[0];
                acc[1] = out[n1];
                acc[2] = out[2 * n1];
            }
            dot_accumulate<OP_>(a, o.b, c, (long long)v, r, acc);
            out[0] = acc[0];
            out[n1] = acc[1];
            out[2 * n1] = acc[2];
        } else {
            pull_store<OP>(pull_out<OP_>(a, o.b, c, (long long)v), n1, r);
        }
    };
#pragma unroll 1
    for (int q = 0; q < kWsV; ++q) voxel(q);
}

// AFF: the affine pull -- no deformation ring; positions from `aff`.
template <int DP, int OP, typename IT, bool AFF>
__global__ void __launch_bounds__(kWsThreads, 1) k_pull_ws(const __grid_constant__ LaunchArgs a,
                                                           const __grid_constant__ TileGrid t,
                                                           const __grid_constant__ CUtensorMap phimap,
                                                           const __grid_constant__ CUtensorMap imgmap,
                                                           const __grid_constant__ AffineMap aff) {
    extern __shared__ __align__(128) float4 smem4[];
    __shared__ __align__(8) unsigned long long bars[kWsStages + 3 * kWsBufs + 2];
    __shared__ Box rec[kWsBufs];
    __shared__ int wrec[2][kWsCons / 32][6];   // per-warp first-tap bounds, by tile parity
    __shared__ volatile int s_abort;
    const Geometry& g = a.g;
    const int G = gridDim.x;
    const int T0 = blockIdx.x;
    if (T0 >= t.ntiles) return;
    const int ntl = (t.ntiles - T0 + G - 1) / G;
    const int nc = g.nc;
    const int D0 = (int)g.d1[0], D1 = (int)g.d1[1], D2 = (int)g.d1[2];
    float* ring = reinterpret_cast<float*>(smem4);
    float* bufs = ring + kWsStages * 3 * kWsNV;
    const unsigned phi_full = smem_addr(&bars[0]);
    const unsigned box_full = smem_addr(&bars[kWsStages]);
    const unsigned box_empty = smem_addr(&bars[kWsStages + kWsBufs]);
    const unsigned bnd_full = smem_addr(&bars[kWsStages + 2 * kWsBufs]);   // two, by tile parity
    const unsigned rec_full = smem_addr(&bars[kWsStages + 2 * kWsBufs + 2]);   // box record published
    // an image TMA cannot address: the consumers load every box themselves, one
    // unit ahead, and publish their bounds two tiles ahead
    const bool ahead = t.img_tma == 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (!AFF && a.sample) {
        if (warp == 0) {
            const bool over = sampled_overflow<DP, OP>(a);
            if (lane == 0) s_abort = over;
        }
        __syncthreads();
        if (s_abort) return;
    }
    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int k = 0; k < kWsStages; ++k) mbar_init(phi_full + 8u * k, 1);
        for (int k = 0; k < kWsBufs; ++k) {
            mbar_init(box_full + 8u * k, 1);
            mbar_init(rec_full + 8u * k, 1);
            mbar_init(box_empty + 8u * k, kWsCons / 32);
        }
        mbar_init(bnd_full, kWsCons / 32);
        mbar_init(bnd_full + 8u, kWsCons / 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp == kWsCons / 32) {
        // ---------------- producer warp ----------------
        auto load_phi = [&](int j) {   // lane 0: tile j's deformation into slot j % kWsStages
            if (!AFF && t.phi_tma && lane == 0) {
                const TileOrigin o = ws_origin(t, T0 + j * G);
                const unsigned bar = phi_full + 8u * (j % kWsStages);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                mbar_expect_tx(bar, (unsigned)(3 * kWsNV * sizeof(float)));
                tma_load_4d(smem_addr(ring + (j % kWsStages) * 3 * kWsNV), &phimap, bar, o.x0, o.y0, o.z0, 3 * o.b);
            }
        };
        for (int j = 0; j < kWsStages && j < ntl; ++j) load_phi(j);
        for (int j = 0; j < ntl && !s_abort; ++j) {
            const TileOrigin o = ws_origin(t, T0 + j * G);
            if (!mbar_wait(bnd_full + 8u * (j & 1), (unsigned)((j >> 1) & 1))) {
                s_abort = 1;
                break;
            }
            Box box = ws_tile_box<DP>(g, t, wrec[j & 1], lane);
            if (box.mode == 1 && !box.tma) {
                // one mode for every channel: a box too large to be loaded row by row
                // stays in shared memory only if all its channels take the window
                Box rows = box;
                ws_async_pitch(rows, g, box.lo[0], box.ext[0] - (box.lo[0] - box.xo));
                if (rows.mode == 2 &&
                    !(g.nbnd == 1 && t.img_tma && ws_mirror_ok(box, g, t, a.bnd.code[0][0], a.bnd.code[0][1], a.bnd.code[0][2])))
                    box.mode = 2;
            }
            for (int c = 0; c < nc; ++c) {
                const int q = j * nc + c, b = q % kWsBufs, k = q / kWsBufs;
                if (k >= 1 && !mbar_wait(box_empty + 8u * b, (unsigned)((k - 1) & 1))) {
                    s_abort = 1;
                    break;
                }
                // the consumers have finished unit q - 2, so every unit of tile
                // j - 2: its ring slot is free for tile j + 2
                if (c == 0 && j >= 2 && j - 2 + kWsStages < ntl) load_phi(j - 2 + kWsStages);
                // interior boxes, and boundary boxes whose margins are mirrors
                // of their own elements (tma = 2: completed by the consumers),
                // arrive by one TMA copy; all others are loaded row by row by the
                // consumers (tma = 3; with DST-II margins, 4: and signed)
                Box ub = box;
                int b0, b1, b2;
                bnd_code(a, c, b0, b1, b2);
                const float* f0 = a.in + ((long long)o.b * nc + c) * g.n0;
                if (ub.mode == 1 && !ub.tma) {
                    if (t.img_tma && ws_mirror_ok(ub, g, t, b0, b1, b2)) {
                        ub.tma = 2;
                        ub.P = kWsWinX;
                        ub.Q = kWsWinX * t.winy;
                        ub.size = kWsCap;
                    } else {
                        ws_async_pitch(ub, g, ub.lo[0], ub.ext[0] - (ub.lo[0] - ub.xo));
                        ub.base = (int)(((long long)(reinterpret_cast<uintptr_t>(f0) >> 2) + ub.lo[0] +
                                         g.d0[0] * (ub.lo[1] + g.d0[1] * (long long)ub.lo[2])) & 3);
                        if ((b0 == 2 && !(ub.interior & 1)) || (b1 == 2 && !(ub.interior & 2)) ||
                            (b2 == 2 && !(ub.interior & 4)))
                            ub.tma = 4;
                    }
                }
                if (lane == 0) {
                    rec[b] = ub;
                    mbar_arrive(rec_full + 8u * b);
                    const unsigned fb = box_full + 8u * b;
                    if (ub.mode == 1 && ub.tma <= 2) {
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        mbar_expect_tx(fb, (unsigned)(kWsWinX * t.winy * t.winz * sizeof(float)));
                        tma_load_4d(smem_addr(bufs + b * kWsCap), &imgmap, fb, ub.xo, ub.lo[1], ub.lo[2], o.b * nc + c);
                    } else {
                        mbar_arrive(fb);
                    }
                }
            }
        }
        return;
    }

    // ---------------- consumer warps ----------------
    // Each warp reduces the first-tap bounds of its voxels of tile j + 1 before
    // it evaluates tile j, so the producer can stage box j + 1 meanwhile.
    const int ctid = threadIdx.x;
    // A deformation TMA cannot address: every thread copies the words of its own
    // voxels, one cp.async group per tile, and waits for its own groups only.
    const bool own_phi = !AFF && !t.phi_tma;
    auto copy_phi = [&](int j) {
        if (j < ntl) {
            const TileOrigin o = ws_origin(t, T0 + j * G);
            float* slot = ring + (j % kWsStages) * 3 * kWsNV;
            const float* phi = a.phi + (long long)o.b * 3 * g.n1;
#pragma unroll
            for (int q = 0; q < kWsV; ++q) {
                const int lin = ctid + q * kWsCons;
                const IT v = ws_index<IT>(o, lin, D0, D1, D2);
                if (v < 0) continue;
#pragma unroll
                for (int k = 0; k < 3; ++k) cp_async4(slot + k * kWsNV + lin, phi + v + k * g.n1);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (own_phi)
        for (int j = 0; j < kWsStages; ++j) copy_phi(j);
    // wait until at most n of this thread's latest cp.async groups are in flight
    auto wait_groups = [&](int n) {
        if (n == 0) asm volatile("cp.async.wait_group 0;" ::: "memory");
        else if (n == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else if (n == 2) asm volatile("cp.async.wait_group 2;" ::: "memory");
        else asm volatile("cp.async.wait_group 3;" ::: "memory");
    };
    // later_groups: groups committed after tile j's deformation (own_phi)
    auto publish_bounds = [&](int j, int later_groups) -> bool {
        const TileOrigin o = ws_origin(t, T0 + j * G);
        const WsPos<AFF> pos{ring + (j % kWsStages) * 3 * kWsNV, &aff};
        if (own_phi) wait_groups(later_groups);
        else if (!AFF && !mbar_wait(phi_full + 8u * (j % kWsStages), (unsigned)((j / kWsStages) & 1))) return false;
        int mn[3], mx[3];
        ws_warp_bounds<DP, IT>(g, o, pos, ctid, D0, D1, D2, mn, mx);
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                wrec[j & 1][warp][k] = mn[k];
                wrec[j & 1][warp][3 + k] = mx[k];
            }
            mbar_arrive(bnd_full + 8u * (j & 1));
        }
        return true;
    };
    if (!publish_bounds(0, 3)) s_abort = 1;
    // load the rows of unit q's box (all consumers) and commit one group
    auto load_unit = [&](int q) {
        const int j = q / nc, c = q - j * nc;
        const Box& box = rec[q % kWsBufs];
        if (box.mode == 1) {
            const TileOrigin o = ws_origin(t, T0 + j * G);
            int b0, b1, b2;
            bnd_code(a, c, b0, b1, b2);
            load_rows<kWsCons, IT>(box_rows(box), g, b0, b1, b2, a.in + ((long long)o.b * nc + c) * g.n0,
                                   bufs + (q % kWsBufs) * kWsCap, ctid);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (ahead) {
        if (ntl > 1 && !publish_bounds(1, 2)) s_abort = 1;
        if (!mbar_wait(rec_full, 0u)) s_abort = 1;
        if (!s_abort) load_unit(0);
    }
    const int nq = ntl * nc;
    for (int j = 0; j < ntl && !s_abort; ++j) {
        const TileOrigin o = ws_origin(t, T0 + j * G);
        const WsPos<AFF> pos{ring + (j % kWsStages) * 3 * kWsNV, &aff};
        // committed after the deformation of the tile whose bounds come next: two
        // later tiles'; ahead: the next tile's and this unit's rows
        const int la = ahead ? 2 : 1;
        if (j + la < ntl && !publish_bounds(j + la, 2)) s_abort = 1;
        if (s_abort) break;
        for (int c = 0; c < nc; ++c) {
            const int q = j * nc + c, b = q % kWsBufs, k = q / kWsBufs;
            if (ahead && q + 1 < nq) {
                const int b1 = (q + 1) % kWsBufs;
                if (!mbar_wait(rec_full + 8u * b1, (unsigned)(((q + 1) / kWsBufs) & 1))) s_abort = 1;
                if (s_abort) break;
                load_unit(q + 1);
            }
            if (!mbar_wait(box_full + 8u * b, (unsigned)(k & 1))) s_abort = 1;
            if (s_abort) break;
            const Box& box = rec[b];
            float* buf = bufs + b * kWsCap;
            if (box.mode == 1 && box.tma >= 2) {   // all consumers load or complete the box
                int b0, b1, b2;
                bnd_code(a, c, b0, b1, b2);
                if (box.tma == 2) {
                    ws_mirror_fixup(box, g, b0, b1, b2, buf, ctid, kWsCons);
                } else {
                    if (!ahead) {
                        load_unit(q);
                        wait_groups(0);
                    } else {
                        // this unit's rows; later: the deformation copied after the
                        // previous tile (first channel), the next unit's rows
                        wait_groups((q + 1 < nq ? 1 : 0) + (own_phi && c == 0 && j > 0 ? 1 : 0));
                    }
                    asm volatile("bar.sync 1, %0;" ::"n"(kWsCons) : "memory");
                    if (box.tma == 4) {
                        sign_rows<kWsCons>(box_rows(box), g, b0, b1, b2, buf, ctid);
                        asm volatile("bar.sync 1, %0;" ::"n"(kWsCons) : "memory");
                    }
                }
            }
            ws_pull_unit<DP, OP, IT>(a, o, ctid, pos, c, box, buf, D0, D1, D2);
            __syncwarp();
            if (lane == 0) mbar_arrive(box_empty + 8u * b);
        }
        if (s_abort) break;
        if (own_phi) copy_phi(j + kWsStages);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// Rows and planes of the image window for tiles that need about ny x nz of them:
// the whole buffer is used, rows in multiples of four (plane pitches that are
// multiples of 32 words) when the planes still fit.  A need beyond the buffer
// keeps the window of an undeformed tile.
void ws_window(TileGrid& t, double ny, double nz) {
    const int y4 = ((int)std::ceil(ny) + 3) & ~3, y1 = (int)std::ceil(ny);
    t.winy = 24;
    t.winz = kWsRows / 24;
    if (!(ny >= 1.0 && nz >= 1.0 && ny <= 256.0 && nz <= 256.0)) return;
    for (int y : {y4, y1})
        if (y <= 256 && kWsRows / y >= nz) {
            t.winy = y;
            t.winz = kWsRows / y < 256 ? kWsRows / y : 256;
            return;
        }
}

// Tile grid of 8 x 16 x 15 tiles over the sample grid (all batches), with the
// multiply-shift constants of ws_origin.
TileGrid ws_make_grid(const LaunchArgs& a) {
    TileGrid t;
    t.lx = 3;
    t.ly = 3;
    t.lz = 4;   // unused here: the z side of a tile is kWsTz
    t.ntx = (int)((a.g.d1[0] + 7) >> 3);
    t.nty = (int)((a.g.d1[1] + kWsTy - 1) >> kWsLy);
    t.ntz = (int)((a.g.d1[2] + kWsTz - 1) / kWsTz);
    t.cap = kWsCap;
    t.ntiles = t.ntx * t.nty * t.ntz * a.g.nb;
    auto magic = [](int d, unsigned long long& m, int& sh) {
        int l = 0;
        while ((1LL << l) < d) ++l;
        sh = 31 + l;
        m = ((1ULL << sh) + (unsigned long long)d - 1) / (unsigned long long)d;
    };
    magic(t.ntx, t.mx, t.sx);
    magic(t.nty, t.my, t.sy);
    magic(t.ntz, t.mz, t.sz);
    t.pmod = 8;
    t.img_tma = t.phi_tma = 0;
    t.nv = kWsNV;
    t.stages = kWsStages;
    // the sample grid usually spans the image: a tile's footprint scales with their
    // ratio, plus the taps and some displacement.  A ratio above the smallest of the
    // three (and above one) is a slab's, which spans a part of the image there.
    const double most = std::fmax(1.0, grid_zoom(a));
    const double ry = a.g.d1[1] > 1 ? (double)(a.g.d0[1] - 1) / (double)(a.g.d1[1] - 1) : 1.0;
    const double rz = a.g.d1[2] > 1 ? (double)(a.g.d0[2] - 1) / (double)(a.g.d1[2] - 1) : 1.0;
    ws_window(t, (kWsTy - 1) * std::fmin(ry, most) + a.g.dp[0] + 3.5, (kWsTz - 1) * std::fmin(rz, most) + a.g.dp[0] + 3.5);
    return t;
}

// 4-D map over the deformation stack (d1, 3 * nb) whose box is one tile's
// three components (8, 16, 15, 3); false when TMA cannot address it.
bool encode_ws_phi_map(CUtensorMap* map, const float* base, const long long d[3], long long planes) {
    EncodeFn fn = encode_fn();
    if (!fn) return false;
    if ((reinterpret_cast<uintptr_t>(base) & 15) || (d[0] & 3)) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)d[0], (cuuint64_t)d[1], (cuuint64_t)d[2], (cuuint64_t)planes};
    for (int k = 0; k < 4; ++k)
        if (dims[k] == 0 || dims[k] > (1ULL << 32)) return false;
    const cuuint64_t strides[3] = {(cuuint64_t)d[0] * 4, (cuuint64_t)(d[0] * d[1]) * 4,
                                   (cuuint64_t)(d[0] * d[1] * d[2]) * 4};
    for (int k = 0; k < 3; ++k)
        if (strides[k] >= (1ULL << 40)) return false;
    const cuuint32_t box[4] = {8, (cuuint32_t)kWsTy, (cuuint32_t)kWsTz, 3};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

// 4-D map over an image stack (d0, d1, d2, planes) with rows of `pitch` elements
// whose box is the image window of t; false when TMA cannot address the image.
bool encode_window_map(CUtensorMap* map, const float* base, const long long d[3], long long pitch, long long planes,
                       const TileGrid& t) {
    auto fn = encode_fn();
    if (!fn) return false;
    if ((reinterpret_cast<uintptr_t>(base) & 15) || (pitch & 3)) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)d[0], (cuuint64_t)d[1], (cuuint64_t)d[2], (cuuint64_t)planes};
    for (int k = 0; k < 4; ++k)
        if (dims[k] == 0 || dims[k] > (1ULL << 32)) return false;
    const cuuint64_t strides[3] = {(cuuint64_t)pitch * 4, (cuuint64_t)(pitch * d[1]) * 4,
                                   (cuuint64_t)(pitch * d[1] * d[2]) * 4};
    for (int k = 0; k < 3; ++k)
        if (strides[k] >= (1ULL << 40)) return false;
    const cuuint32_t box[4] = {(cuuint32_t)kWsWinX, (cuuint32_t)t.winy, (cuuint32_t)t.winz, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

// Rows of n floats copied to rows of `pitch` floats (the padding stays as it is).
__global__ void __launch_bounds__(256) k_pad_rows(const float* __restrict__ in, float* __restrict__ out, unsigned n,
                                                  unsigned pitch, unsigned rows) {
    const unsigned lane = threadIdx.x & 31;
    for (unsigned r = blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8) {
        const float* src = in + (size_t)r * n;
        float* dst = out + (size_t)r * pitch;
        for (unsigned x = lane; x < n; x += 32) dst[x] = __ldg(src + x);
    }
}

// Image of a launch as TMA reads it: the caller's, or a copy with its rows padded
// to 16 bytes when the caller's rows are not multiples of that.  The copy moves
// 8 bytes per image voxel and channel (28 MB of image: about 10 us) and saves the
// consumers loading every box themselves (181x217x181 cubic pull, GB300: 186 us
// with it, 279 us without).  It is not made for images much larger than the
// sample grid, above kScratchMost, or while the stream is being captured into a graph.
struct WsImage {
    float* copy = nullptr;
    bool tma = false;
};

inline cudaError_t ws_image(const LaunchArgs& a, const TileGrid& t, CUtensorMap* map, WsImage& im, cudaStream_t s) {
    const Geometry& g = a.g;
    const long long planes = (long long)g.nc * g.nb;
    im.tma = encode_window_map(map, a.in, g.d0, g.d0[0], planes, t);
    if (im.tma) return cudaSuccess;
    const long long pitch = (g.d0[0] + 3) & ~3LL, rows = g.d0[1] * g.d0[2] * planes;
    const long long bytes = pitch * rows * 4;
    if (g.n0 > 4 * g.n1 || bytes > (long long)kScratchMost || rows > 0x7fffffffLL) return cudaSuccess;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
        (void)cudaGetLastError();
        return cudaSuccess;
    }
    if (scratch_alloc(reinterpret_cast<void**>(&im.copy), (size_t)bytes, s) != cudaSuccess) {
        (void)cudaGetLastError();   // no memory for the copy: the consumers load the boxes
        im.copy = nullptr;
        return cudaSuccess;
    }
    const long long want = (rows + 7) / 8, cap_grid = 16LL * sm_count();
    k_pad_rows<<<(unsigned)(want < cap_grid ? want : cap_grid), 256, 0, s>>>(a.in, im.copy, (unsigned)g.d0[0],
                                                                            (unsigned)pitch, (unsigned)rows);
    const cudaError_t e = cudaGetLastError();
    im.tma = e == cudaSuccess && encode_window_map(map, im.copy, g.d0, pitch, planes, t);
    return e;
}

// CTAs of a launch (CTA c takes tiles c, c + G, ...).  Where G and the tiles along x
// share a factor, a CTA meets the same few x positions again and again, and the tiles
// at the border of the image, whose boxes do not arrive by TMA alone, all fall on some
// of the CTAs.  So a G without a common factor, unless it takes one more round of
// tiles.  GB300, 152 SMs, cubic pull: 192^3 152 CTAs 152 us, 151 142; bounds (0, 1, 2)
// 175 / 146; 160x192x160 quadratic, bounds (0, 1, 2) 87 / 78.  (The push kernels gain
// too, 192^3 228 / 224 us, but a contracted 256^3 x 3 loses, 1584 / 1623: they keep
// all their CTAs.)
inline int ws_grid(const TileGrid& t) {
    const int want = sm_count();
    if (t.ntiles < 2 * want) return t.ntiles < want ? t.ntiles : want;
    const int rounds = (t.ntiles + want - 1) / want;
    for (int g = want; g > want - 8 && g > 1 && (t.ntiles + g - 1) / g == rounds; --g) {
        int x = g, y = t.ntx;
        while (y) {
            const int r = x % y;
            x = y;
            y = r;
        }
        if (x == 1) return g;
    }
    return want;
}

template <int DP, int OP, typename IT, bool AFF>
cudaError_t launch_ws_one(const LaunchArgs& a, const TileGrid& t, const CUtensorMap& phimap, const AffineMap& aff,
                          cudaStream_t s) {
    CUtensorMap imgmap;
    std::memset(&imgmap, 0, sizeof imgmap);
    TileGrid tt = t;
    auto kern = k_pull_ws<DP, OP, IT, AFF>;
    cudaError_t e = opt_in(kern, kWsSmem);
    if (e != cudaSuccess) return e;
    WsImage im;
    e = ws_image(a, t, &imgmap, im, s);
    if (e == cudaSuccess) {
        tt.img_tma = im.tma ? 1 : 0;
        kern<<<ws_grid(tt), kWsThreads, kWsSmem, s>>>(a, tt, phimap, imgmap, aff);
        e = cudaGetLastError();
    }
    if (im.copy) {
        const cudaError_t ef = cudaFreeAsync(im.copy, s);
        if (e == cudaSuccess) e = ef;
    }
    return e;
}

template <int OP, typename IT, bool AFF = false>
cudaError_t ws_dispatch(const LaunchArgs& a, const TileGrid& t, const CUtensorMap& phimap, cudaStream_t s,
                        const AffineMap& aff = AffineMap{}) {
    switch (a.g.dp[0]) {
        case 1: return launch_ws_one<1, OP, IT, AFF>(a, t, phimap, aff, s);
        case 2: return launch_ws_one<2, OP, IT, AFF>(a, t, phimap, aff, s);
        case 3: return launch_ws_one<3, OP, IT, AFF>(a, t, phimap, aff, s);
        case 4: return launch_ws_one<4, OP, IT, AFF>(a, t, phimap, aff, s);
        default: return launch_ws_one<5, OP, IT, AFF>(a, t, phimap, aff, s);
    }
}

// One op of the warp-specialised family on 32-bit or 64-bit voxel indices.
template <int OP>
cudaError_t ws_dispatch_op(const LaunchArgs& a, const TileGrid& t, const CUtensorMap& phimap, cudaStream_t s) {
    const bool small = a.g.n0 < (1LL << 31) - 1 && a.g.n1 < (1LL << 31) - 1;
    return small ? ws_dispatch<OP, int>(a, t, phimap, s) : ws_dispatch<OP, long long>(a, t, phimap, s);
}

}  // namespace
}  // namespace pp
