// pp_push.cuh -- tiled push family: push, push_grad and the affine push.
//
// Included by pp_tiled_push.cu, pp_tiled_pushg.cu and pp_tiled_affine.cu.
//
// A CTA walks tiles of 2^lx x 2^ly x 2^lz sample voxels.  Every tile scatters
// its weighted taps into a shared-memory accumulator that covers the tile's
// footprint box in the image and flushes the box with 4-wide global reductions.
//
// Accumulator: two 32-bit fixed-point words per element, filled by shared-memory
// integer reductions, which run at one wavefront per clock on this part and are what
// bounds the scatter.  A contribution is formed in float32 and split: its upper part
// in quanta of 2^(E - 22), the rest in quanta of 2^(E - 43).  The scale follows the
// largest value of the tile and the sum of all, whichever needs more (push_exponent), so
// that the quantum is at most 2^-41 of the largest value.
// (One word per element, bounded by a first pass over the tile, takes 226 us at 192^3
// cubic where two take 331; but 31 bits below the largest sum of a tile leave the
// elements of its dark parts, of the sample grid's edge and of contracted tiles with
// errors an order of magnitude above float32's, and push_grad of noise with 1.45e-7
// against 1.1e-7 in the l2 norm.  It was taken back.)
//
// Lanes: a warp covers 2^lx voxels in x and 32 / 2^lx rows.  The row pitch is an odd
// multiple of 2^lx and the plane pitch a multiple of 32, so that a first tap one
// row or plane off its neighbours' does not change its bank: of the pitches
// tried on a smooth +-5 voxel field, 32-wide tiles with both pitches multiples
// of 32 gave 2.0 wavefronts per reduction, 16 x 2 lanes 2.2, 8 x 4 lanes 2.3,
// and pitches without that property 2.8 to 3.4.
#pragma once

#include <type_traits>

#include "pp_tiled_impl.cuh"

namespace pp {
namespace {

// Four CTAs of 128 threads per SM rather than two of 256: the phases of a tile (bounds,
// scatter, flush) are separated by barriers, and more CTAs in different phases keep the
// shared-memory pipe busy (cubic 192^3, best tile of each, us: 335 against 345; three of
// 128 388, five 334; push_grad 181x217x181 394 against 457, 418, 397).
constexpr int kPushThreads = 128;
constexpr int kPushCtas = 4;
constexpr int kFarTap = 1 << 22;    // first taps beyond this leave float32 weights inexact: per-voxel path

// Voxel `lin` of a tile (x fastest) -> its sample index within the batch.
// full: the whole tile lies inside the sample grid.
struct PushTile {
    int x0, y0, z0, D0, D1, D2, lx, ly;
    bool full;
    __device__ __forceinline__ PushTile(const TileOrigin& o, const TileGrid& t, const Geometry& g)
        : x0(o.x0), y0(o.y0), z0(o.z0), D0((int)g.d1[0]), D1((int)g.d1[1]), D2((int)g.d1[2]), lx(t.lx), ly(t.ly),
          full(o.x0 + (1 << t.lx) <= (int)g.d1[0] && o.y0 + (1 << t.ly) <= (int)g.d1[1] &&
               o.z0 + (1 << t.lz) <= (int)g.d1[2]) {}
    __device__ __forceinline__ void coords(int lin, int& x, int& y, int& z) const {
        x = x0 + (lin & ((1 << lx) - 1));
        y = y0 + ((lin >> lx) & ((1 << ly) - 1));
        z = z0 + (lin >> (lx + ly));
    }
    __device__ __forceinline__ bool inside(int lin) const {
        if (full) return true;
        int x, y, z;
        coords(lin, x, y, z);
        return x < D0 && y < D1 && z < D2;
    }
    // voxels of the tile that lie inside the sample grid
    __device__ __forceinline__ int count(const TileGrid& t) const {
        return full ? t.nv
                    : min(1 << t.lx, D0 - x0) * min(1 << t.ly, D1 - y0) * min(1 << t.lz, D2 - z0);
    }
    template <typename IT>
    __device__ __forceinline__ IT index(int lin) const {
        int x, y, z;
        coords(lin, x, y, z);
        return (IT)x + (IT)D0 * ((IT)y + (IT)D1 * (IT)z);
    }
};

// Sample position of voxel `lin`: x = phi - 1 from the ring slot, or (AFF)
// A * (i, j, k, 1) from its grid coordinates; with the validity test.
template <bool AFF>
struct PushPos {
    const float* slot;
    int nv;
    const AffineMap* A;
    __device__ __forceinline__ bool operator()(const Geometry& g, const PushTile& pt, int lin, float& x0, float& x1,
                                               float& x2) const {
        if constexpr (AFF) {
            int x, y, z;
            pt.coords(lin, x, y, z);
            affine_position(*A, (float)x, (float)y, (float)z, x0, x1, x2);
            return position_valid(x0, x1, x2, g);
        } else {
            return load_valid(slot[lin], slot[nv + lin], slot[2 * nv + lin], g, x0, x1, x2);
        }
    }
};

// Order-preserving integer image of a float (for integer min / max reductions).
__device__ __forceinline__ int float_key(float v) {
    const int b = __float_as_int(v);
    return b ^ ((b >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float key_float(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }

// Footprint box of a tile in the accumulator (the same in every thread).
struct PushBox {
    int lo[3], e[3];    // minima of the first taps; extents
    int P, Q, size;     // row and plane pitch; words, base offset included
    int mode;           // 0 no valid voxel, 1 accumulator, 2 per-voxel global
    int xin, yin, zin;  // inside the image along each dimension
    int cells;          // > 0: contracted tile, first-tap cells of the box (cell_scatter)
    int group;          // contracted tile: kCellChannels channels at once
    int vec;            // the box has the image's 16-byte alignment
};

// Block-wide minima, maxima, sum and maximum: one record per warp, which every
// warp combines (in the same order), so the results are uniform after one barrier.
// bounds: the minima and maxima too.
__device__ __forceinline__ void tile_combine(int (&wrec)[kPushThreads / 32][8], bool bounds, int (&mn)[3], int (&mx)[3],
                                             float& ssum, float& smax) {
    constexpr int NW = kPushThreads / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (bounds) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            mn[k] = __reduce_min_sync(0xffffffffu, mn[k]);
            mx[k] = __reduce_max_sync(0xffffffffu, mx[k]);
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) ssum += __shfl_xor_sync(0xffffffffu, ssum, d);
    smax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(smax)));
    if (lane == 0) {
        if (bounds) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                wrec[warp][k] = mn[k];
                wrec[warp][3 + k] = mx[k];
            }
        }
        wrec[warp][6] = __float_as_int(ssum);
        wrec[warp][7] = __float_as_int(smax);
    }
    __syncthreads();
    const int* r = wrec[lane & (NW - 1)];
    if (bounds) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            mn[k] = __reduce_min_sync(0xffffffffu, r[k]);
            mx[k] = __reduce_max_sync(0xffffffffu, r[3 + k]);
        }
    }
    ssum = __int_as_float(r[6]);
#pragma unroll
    for (int d = NW / 2; d > 0; d >>= 1) ssum += __shfl_xor_sync(0xffffffffu, ssum, d);
    smax = __uint_as_float(__reduce_max_sync(0xffffffffu, (unsigned)r[7]));
}

// Position bounds of a tile (float_key images; the first tap is monotone in the
// position) -> the box's place and extents.  True: mode 2 is set, pitches to
// follow; false: no valid voxel (mode 0), or coordinates the accumulator does not
// take (mode 2).
template <int DP>
__device__ __forceinline__ bool box_place(int (&mn)[3], int (&mx)[3], const Geometry& g, PushBox& box) {
    box.mode = 0;
    box.cells = 0;
    box.size = 0;
    if (mn[0] > mx[0]) return false;
    box.mode = 2;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        mn[k] = first_tap32(key_float(mn[k]), DP);
        mx[k] = first_tap32(key_float(mx[k]), DP);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (!(mn[k] > -kFarTap && mx[k] < kFarTap && mx[k] - mn[k] < 4096)) return false;
        box.lo[k] = mn[k];
        box.e[k] = mx[k] - mn[k] + DP;
    }
    box.xin = mn[0] >= 0 && mx[0] + DP <= g.d0[0];
    box.yin = mn[1] >= 0 && mx[1] + DP <= g.d0[1];
    box.zin = mn[2] >= 0 && mx[2] + DP <= g.d0[2];
    return true;
}

// Conflict-free pitches of the box when they fit `cap` words, tight ones when only
// those do (mode 1), else mode 2.
__device__ __forceinline__ void box_pitches(const TileGrid& t, int cap, const Geometry& g, PushBox& box) {
    // an odd multiple of the lanes' width in x: their rows start in distinct banks
    long long P = box.e[0] + 3;
    P += (t.pmod - P) & (t.pmod ? 2 * t.pmod - 1 : 31);
    long long Q = P * box.e[1];
    Q += -Q & 31;
    if (Q * box.e[2] + 8 > cap) {      // pack tightly when the padding does not fit
        P = (box.e[0] + 6) & ~3;
        Q = P * box.e[1];
    }
    const bool fits = Q * box.e[2] + 8 <= cap;
    box.size = fits ? (int)((Q * box.e[2] + 7) & ~3LL) : 0;
    box.P = fits ? (int)P : 0;
    box.Q = fits ? (int)Q : 0;
    box.mode = fits ? 1 : 2;
    box.vec = fits && (g.d0[0] & 3) == 0 && ((P | Q) & 3) == 0;
}

// First word of the box in the accumulator of a channel at f0: the image's
// 16-byte alignment where the pitches share it.
__device__ __forceinline__ int box_base(const PushBox& box, const Geometry& g, const float* f0) {
    const long long org = box.lo[0] + g.d0[0] * (box.lo[1] + g.d0[1] * (long long)box.lo[2]);
    return box.vec ? (int)(((long long)(reinterpret_cast<uintptr_t>(f0) >> 2) + org) & 3) : 0;
}

// Add the accumulator box into one channel of the image and clear it.  Four
// consecutive elements of a row that are 16-byte aligned in the image go as one
// 4-wide reduction.  VEC: the box has the image's alignment (image extents a
// multiple of 4), so the accumulator words come and are cleared 16 bytes at a
// time.  Otherwise word by word, lanes of neighbouring rows starting at
// different words of their group so that they read different banks.
// ld4 / ld1 return the value of words w (.. w + 3) and clear them.
template <bool VEC, typename IT, class LD4, class LD1>
__device__ __forceinline__ void push_flush_rows(const PushBox& box, const Geometry& g, int b0, int b1, int b2,
                                                float* f0, int base0, LD4 ld4, LD1 ld1) {
    const int ey = box.e[1], ez = box.e[2], e0 = box.e[0];
    const int dx = (int)g.d0[0];
    RowWalk<kPushThreads> rw((e0 + 6) >> 2, ey);     // groups of 4 that a row can touch
    const IT sy = (IT)g.d0[0];
    const IT sz = (IT)(g.d0[0] * g.d0[1]);
    const int rot = rw.sub & 3;
    for (; rw.rz < ez; rw.next()) {
        const int rz = rw.rz, ry = rw.ry;
        float s = 1.f;
        IT gy = (IT)(box.lo[1] + ry), gz = (IT)(box.lo[2] + rz);
        if (!(box.yin && box.zin)) {
            float sgy, sgz;
            gy = (IT)fold_tap(b1, (long long)box.lo[1] + ry, g.d0[1], sgy);
            gz = (IT)fold_tap(b2, (long long)box.lo[2] + rz, g.d0[2], sgz);
            s = sgy * sgz;
        }
        float* grow = f0 + (gz * sz + gy * sy);
        const int s0 = base0 + rz * box.Q + ry * box.P;
        const int mis = (int)(((reinterpret_cast<uintptr_t>(grow) >> 2) + box.lo[0]) & 3);
        for (int e = 4 * rw.e0 - mis; e < e0; e += 4 << rw.lg) {
            float4 v;
            if constexpr (VEC) {
                v = ld4(s0 + e);
            } else {
                float r[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int eu = e + ((u + rot) & 3);
                    r[u] = eu >= 0 && eu < e0 ? ld1(s0 + eu) : 0.f;
                }
                // r[u] is word (u + rot) mod 4 of the group
                const bool o1 = rot & 1, o2 = rot & 2;
                const float t0 = o1 ? r[3] : r[0], t1 = o1 ? r[0] : r[1], t2 = o1 ? r[1] : r[2], t3 = o1 ? r[2] : r[3];
                v = make_float4(o2 ? t2 : t0, o2 ? t3 : t1, o2 ? t0 : t2, o2 ? t1 : t3);
            }
            if (v.x == 0.f && v.y == 0.f && v.z == 0.f && v.w == 0.f) continue;
            v.x *= s;
            v.y *= s;
            v.z *= s;
            v.w *= s;
            const int gx = box.lo[0] + e;
            if (gx >= 0 && gx + 4 <= dx) {
                atomicAdd(reinterpret_cast<float4*>(grow + gx), v);
            } else {
                const float vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (vv[u] == 0.f) continue;   // also the words before and after the row
                    float sgx;
                    const IT fx = (IT)fold_tap(b0, (long long)gx + u, g.d0[0], sgx);
                    atomicAdd(grow + fx, sgx * vv[u]);
                }
            }
        }
    }
}

template <typename IT, class LD4, class LD1>
__device__ __forceinline__ void push_flush(const PushBox& box, const Geometry& g, int b0, int b1, int b2, float* f0,
                                           int base0, LD4 ld4, LD1 ld1) {
    if (box.vec) push_flush_rows<true, IT>(box, g, b0, b1, b2, f0, base0, ld4, ld1);
    else push_flush_rows<false, IT>(box, g, b0, b1, b2, f0, base0, ld4, ld1);
}

// Exponent E of the accumulator's scale for a tile whose contributions are at most M
// each and S in sum (absolute values): the upper quantum is 2^(E - 22), the lower
// 2^(E - 43).  An upper part is at most 2^22 quanta (E >= log2 M) and an element's
// sum of them at most 2^30 (E >= log2 S - 8); a lower part is at most 2^20 quanta
// and an element receives one per voxel, of which a tile has at most 2^10.  INT_MIN:
// S outside the range the scale factors cover, the tile accumulates in float.
__device__ __forceinline__ int push_exponent(float S, float M) {
    const int es = scale_exponent(S);
    if (es == INT_MIN || es == INT_MAX) return INT_MIN;
    const int em = scale_exponent(M);      // (INT_MIN below 2^-80)
    return max(max(em, es - 8), -80);
}

// Wait until at most n (0..3) of this thread's latest cp.async groups are in flight.
__device__ __forceinline__ void wait_groups(int n) {
    if (n >= 3) asm volatile("cp.async.wait_group 3;\n" ::: "memory");
    else if (n == 2) asm volatile("cp.async.wait_group 2;\n" ::: "memory");
    else if (n == 1) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// Fill ring slot (j mod stages) with tile T: the deformation (not AFF) and
// NVAL components of channel 0 of `vals`.  TMA: thread 0 issues one bulk tensor copy
// per tensor.  Otherwise every thread copies the words it will read itself with
// 4-byte cp.async and commits one group, so no thread waits for another's.
template <int NVAL, bool TMA, typename IT, bool AFF>
__device__ __forceinline__ void push_ring_fill(float* base, int slot_floats, int stages, unsigned bars, int j, int T,
                                               bool live, const LaunchArgs& a, const float* vals, const TileGrid& t,
                                               const CUtensorMap& phimap, const CUtensorMap& valmap) {
    const int nv = t.nv, sidx = j % stages;
    constexpr int NPHI = AFF ? 0 : 3;
    float* slot = base + sidx * slot_floats;
    if constexpr (TMA) {
        if (live && threadIdx.x == 0) {
            const TileOrigin o = tile_origin(t, T);
            const unsigned bar = bars + 8u * sidx;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_expect_tx(bar, (unsigned)((NPHI + NVAL) * nv * sizeof(float)));
            if constexpr (!AFF) tma_load_4d(smem_addr(slot), &phimap, bar, o.x0, o.y0, o.z0, 3 * o.b);
            tma_load_4d(smem_addr(slot + NPHI * nv), &valmap, bar, o.x0, o.y0, o.z0, NVAL * a.g.nc * o.b);
        }
    } else {
        if (live) {
            const TileOrigin o = tile_origin(t, T);
            const PushTile pt(o, t, a.g);
            const long long n1 = a.g.n1;
            const float* phi = AFF ? nullptr : a.phi + (long long)o.b * 3 * n1;
            const float* val = vals + (long long)o.b * a.g.nc * NVAL * n1;
#pragma unroll 2
            for (int lin = threadIdx.x; lin < nv; lin += kPushThreads) {
                if (!pt.inside(lin)) continue;
                const IT v = pt.index<IT>(lin);
                if constexpr (!AFF) {
#pragma unroll
                    for (int k = 0; k < 3; ++k) cp_async4(slot + k * nv + lin, phi + v + k * n1);
                }
#pragma unroll
                for (int k = 0; k < NVAL; ++k) cp_async4(slot + (NPHI + k) * nv + lin, val + v + k * n1);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
}

// Scatter one channel of a tile (values at vslot, NCOMP planes of the tile's
// voxels; ssum, smax: block-wide sum and maximum of their absolute values) into the
// accumulator and add it to the image at f0.  The accumulator is zero before and
// after; the caller synchronises the block before either is used again.
template <int DP, int OP, typename IT, class POS>
__device__ __forceinline__ void push_channel(const Geometry& g, const TileGrid& t, const PushTile& pt, const POS& pos,
                                             const float* vslot, const PushBox& box, int b0, int b1, int b2, float* f0,
                                             float* accf, float ssum, float smax) {
    constexpr int ORD = OP == kPushGrad ? 1 : 0;
    constexpr int NCOMP = OP == kPushGrad ? 3 : 1;
    if (smax == 0.f) return;   // every value of this channel is zero or skipped
    const int nv = t.nv, half = box.size;
    int* acc = reinterpret_cast<int*>(accf);
    const int bxo = box.lo[0], by0 = box.lo[1], bz0 = box.lo[2];
    const unsigned P4 = 4u * box.P, Q4 = 4u * box.Q;
    const int base0 = box_base(box, g, f0);
    const unsigned cbase = smem_addr(accf) + 4u * base0;
    const int E = push_exponent(NCOMP == 3 ? 2.f * ssum : ssum, NCOMP == 3 ? 2.f * smax : smax);
    auto scatter = [&](float sc, auto fixed) {
#pragma unroll 1
        for (int lin = threadIdx.x; lin < nv; lin += kPushThreads) {
            float x0, x1, x2, val[3] = {0.f, 0.f, 0.f};
            if (!pt.inside(lin) || !pos(g, pt, lin, x0, x1, x2)) continue;
            bool fin = true;
#pragma unroll
            for (int p = 0; p < NCOMP; ++p) {
                val[p] = vslot[p * nv + lin];
                fin = fin & finitef(val[p]);
            }
            if (!fin) continue;
            W3<DP, ORD> wx, wy, wz;
            const int ox = spline_taps32<DP, ORD>(x0, wx.w, wx.dw, wx.hw) - bxo;
            const int oy = spline_taps32<DP, ORD>(x1, wy.w, wy.dw, wy.hw) - by0;
            const int oz = spline_taps32<DP, ORD>(x2, wz.w, wz.dw, wz.hw) - bz0;
            push_scatter<DP, OP, decltype(fixed)::value>(wx, wy, wz, val[0] * sc, val[1] * sc, val[2] * sc,
                                                         cbase + 4u * (unsigned)(oz * box.Q + oy * box.P + ox), P4, Q4,
                                                         4u * half);
        }
        __syncthreads();
    };
    if (E != INT_MIN) {
        scatter(pow2f(22 - E), std::true_type{});
        const float q1 = pow2f(E - 22), q2 = pow2f(E - 43);
        auto val = [&](int h, int l) { return fmaf((float)h, q1, (float)l * q2); };
        push_flush<IT>(box, g, b0, b1, b2, f0, base0, [&](int w) {
            int4* hp = reinterpret_cast<int4*>(acc + w);
            int4* lp = reinterpret_cast<int4*>(acc + half + w);
            const int4 h = *hp, l = *lp;
            *hp = *lp = make_int4(0, 0, 0, 0);
            return make_float4(val(h.x, l.x), val(h.y, l.y), val(h.z, l.z), val(h.w, l.w));
        }, [&](int w) {
            const int h = acc[w], l = acc[half + w];
            acc[w] = acc[half + w] = 0;
            return val(h, l);
        });
    } else {
        scatter(1.f, std::false_type{});
        push_flush<IT>(box, g, b0, b1, b2, f0, base0, [&](int w) {
            const float4 v = *reinterpret_cast<const float4*>(accf + w);
            *reinterpret_cast<float4*>(accf + w) = make_float4(0.f, 0.f, 0.f, 0.f);
            return v;
        }, [&](int w) {
            const float v = accf[w];
            accf[w] = 0.f;
            return v;
        });
    }
}

// ---- contracted tiles ---------------------------------------------------------
//
// A tile with several samples per first-tap cell (a contracting deformation) is
// scattered cell by cell.  The voxels of a batch are counting-sorted by cell;
// then a warp takes a cell, one tap (or two) per lane, sums the cell's voxels in
// registers for up to three channels at once, a few voxels at a time, and adds each
// tap's sums to the two-word accumulator.  A voxel costs the warp its position within the
// cell and its values (16-byte broadcast loads of two voxels) and packed f32x2
// arithmetic: the lane's weights are polynomials in that position whose
// coefficients the lane holds.
// A cell's sums are float32: 32 voxels (two halves of 16) between fixed-point additions
// keep their rounding near that of the terms themselves (cubic, contracted 0.25x, l2
// error against 64 bits of push of noise / push_grad of noise, 1e-7: halves of 8 1.29 /
// 1.35, of 16 1.36 / 1.42, of any length 1.45 / 1.52; every voxel into fixed point by
// itself 1.67 / 1.47; us, 192^3: 489, 471, 462, 618).
// From three samples per cell on (cubic push; push_grad four, quadratic six) this is the
// faster scatter.  192^3, one channel, us, cell by cell / per voxel: 0.35x 441 / 614,
// 0.5x 480 / 560, 0.6x 544 / 454; quadratic 0.4x 367 / 332; push_grad 160^3 0.4x 349 / 417,
// 0.5x 402 / 340.
constexpr int kCellBatch = 512;       // voxels sorted at a time
constexpr int kCellRun = 16;          // pairs of voxels a lane sums before they go into fixed point
template <int DP, int OP>             // samples per cell from which a tile counts as contracted
constexpr int kCellMin = DP == 3 ? 6 : (OP == kPush ? 3 : 4);
constexpr int kCellChannels = 3;      // channels summed at once (push)

__device__ __forceinline__ float2 dup(float v) { return make_float2(v, v); }

// One lane's weight (and derivative) along an axis, for two voxels at once, in the
// factored form of spline_weights (a power basis in s cancels where a weight is
// small).  u is the position from the end of the spline's piece that makes the piece
// one of two shapes: degree 3 u^3 / 6 and c - u^2 + u^3 / 2 with u = s or 1 - s,
// degree 2 u^2 / 2 with u = 1/2 + s or 1/2 - s and 3/4 - s^2.
template <int DP, int ORD>
struct LanePoly {
    float2 sg, off, k3, k2, c, cl, m2, m1;
    __device__ __forceinline__ void set(int i) {
        if constexpr (DP == 4) {
            const bool mirror = i == 0 || i == 2, outer = i == 0 || i == 3;
            const float s1 = mirror ? -1.f : 1.f;
            constexpr float c6 = 1.0f / 6.0f, c23 = 2.0f / 3.0f;
            sg = dup(s1);
            off = dup(mirror ? 1.f : 0.f);
            k3 = dup(outer ? c6 : 0.5f);
            k2 = dup(outer ? 0.f : -1.f);
            // 2/3 in two words: rounded to one it is off by 2e-8, in one direction for every sample
            c = dup(outer ? 0.f : c23);
            cl = dup(outer ? 0.f : (float)(2.0 / 3.0 - (double)c23));
            m2 = dup(s1 * (outer ? 0.5f : 1.5f));
            m1 = dup(outer ? 0.f : -2.f * s1);
        } else {
            sg = dup(i == 0 ? -1.f : 1.f);
            off = dup(i == 1 ? 0.f : 0.5f);
            k2 = dup(i == 1 ? -1.f : 0.5f);
            c = dup(i == 1 ? 0.75f : 0.f);
            m1 = dup(i == 0 ? -1.f : (i == 1 ? -2.f : 1.f));
        }
    }
    __device__ __forceinline__ float2 at(float2 s) const { return __ffma2_rn(s, sg, off); }
    __device__ __forceinline__ float2 val(float2 u) const {
        if constexpr (DP == 4) return __fadd2_rn(c, __ffma2_rn(__fmul2_rn(u, u), __ffma2_rn(u, k3, k2), cl));
        else return __ffma2_rn(__fmul2_rn(u, k2), u, c);
    }
    __device__ __forceinline__ float2 der(float2 u) const {
        if constexpr (DP == 4) return __fmul2_rn(u, __ffma2_rn(u, m2, m1));
        else return __fmul2_rn(u, m1);
    }
};

// Position within the cell, as spline_weights measures it.
template <int DP>
__device__ __forceinline__ float cell_position(float x, float fo) {
    return __fsub_rn(x, fo + 1.0f);
}

// Shared-memory layout of the sorted voxels: pairs of voxels (2t, 2t + 1) as
// 16-byte rows (sx, sx', sy, sy'), (sz, sz', a, a') and, when there is more than
// one value per voxel, (b, b', c, c').
struct CellArrays {
    float4 *A, *B, *C;
    unsigned* tag;       // cell << 16 | rank of every voxel of the batch (all ones: skipped)
    int* start;          // per cell: count, then first sorted position
};

// Sum every cell's voxels and add the sums to the accumulators (NVAL words
// arrays of two words per element, `half` words apart).  Warps take cells in turn.
template <int DP, int OP, int NVAL>
__device__ __forceinline__ void cell_scatter(const CellArrays& ca, int ncells, int c0, int c01, unsigned acc, int P,
                                             int Q, int half, const float* inv, const int* base0) {
    constexpr int ORD = OP == kPushGrad ? 1 : 0;
    constexpr int PASSES = DP == 4 ? 2 : 1;
    constexpr int NOUT = OP == kPushGrad ? 1 : NVAL;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tt = lane < DP * DP * DP ? lane : 0;
    const int ti = tt % DP, tj = (tt / DP) % DP, tk = tt / (DP * DP);
    LanePoly<DP, ORD> px, py, pz[PASSES];
    px.set(ti);
    py.set(tj);
#pragma unroll
    for (int p = 0; p < PASSES; ++p) pz[p].set(tk + 2 * p);
    const int off = ti + P * tj + Q * tk;
    const bool live = DP == 4 || lane < DP * DP * DP;
    for (int cell = warp; cell < ncells; cell += kPushThreads / 32) {
        const int b = ca.start[cell] >> 1, e = ca.start[cell + 1] >> 1;
        // cell -> box element of its first tap
        const int cz = cell / c01, cr = cell - cz * c01, cy = cr / c0, cx = cr - cy * c0;
        const unsigned base = acc + 4u * (unsigned)(cx + P * cy + Q * cz + off);
        for (int t0 = b; t0 < e; t0 += kCellRun) {
            const int t1 = min(t0 + kCellRun, e);
            float2 acc2[PASSES][NOUT];
#pragma unroll
            for (int p = 0; p < PASSES; ++p)
#pragma unroll
                for (int c = 0; c < NOUT; ++c) acc2[p][c] = make_float2(0.f, 0.f);
#pragma unroll 2
            for (int t = t0; t < t1; ++t) {
                const float4 a4 = ca.A[t], b4 = ca.B[t];
                const float2 ux = px.at(make_float2(a4.x, a4.y)), uy = py.at(make_float2(a4.z, a4.w));
                const float2 sz = make_float2(b4.x, b4.y);
                float2 v[3];
                v[0] = make_float2(b4.z, b4.w);
                if constexpr (NVAL > 1) {
                    const float4 c4 = ca.C[t];
                    v[1] = make_float2(c4.x, c4.y);
                    v[2] = make_float2(c4.z, c4.w);
                }
                const float2 wx = px.val(ux), wy = py.val(uy);
                if constexpr (OP == kPushGrad) {
                    // v0 dwx wy wz + v1 wx dwy wz + v2 wx wy dwz
                    const float2 f = __ffma2_rn(wy, __fmul2_rn(v[0], px.der(ux)),
                                                __fmul2_rn(py.der(uy), __fmul2_rn(v[1], wx)));
                    const float2 h = __fmul2_rn(wy, __fmul2_rn(v[2], wx));
#pragma unroll
                    for (int p = 0; p < PASSES; ++p) {
                        const float2 uz = pz[p].at(sz);
                        acc2[p][0] = __fadd2_rn(acc2[p][0], __ffma2_rn(pz[p].val(uz), f, __fmul2_rn(pz[p].der(uz), h)));
                    }
                } else {
                    const float2 wxy = __fmul2_rn(wx, wy);
#pragma unroll
                    for (int p = 0; p < PASSES; ++p) {
                        const float2 w = __fmul2_rn(wxy, pz[p].val(pz[p].at(sz)));
#pragma unroll
                        for (int c = 0; c < NOUT; ++c) acc2[p][c] = __ffma2_rn(w, v[c], acc2[p][c]);
                    }
                }
            }
            if (live) {
#pragma unroll
                for (int p = 0; p < PASSES; ++p)
#pragma unroll
                    for (int c = 0; c < NOUT; ++c) {
                        // y in units of the upper quantum, |y| <= 2^22: hi = round(y), lo = round((y - hi) * 2^21)
                        const float y = (acc2[p][c].x + acc2[p][c].y) * inv[c];
                        const float t1f = __fadd_rn(y, kMagic);
                        const float r = __fsub_rn(y, __fsub_rn(t1f, kMagic));
                        const unsigned ad = base + 4u * (unsigned)(2 * p * Q + c * 2 * half + base0[c]);
                        red_s32_nb(ad, __float_as_int(t1f) - kMagicBits);
                        red_s32_nb(ad + 4u * half, __float_as_int(__fmaf_rn(r, kLoScale, kMagic)) - kMagicBits);
                    }
            }
        }
    }
}

// Persistent push family.  CTA i walks tiles i, i + G, ...; the ring holds the
// next tiles' deformation and channel-0 values.
// AFF: the affine push -- positions A * (i, j, k, 1) from `aff`, no deformation.
template <int DP, int OP, typename IT, bool TMA, bool AFF>
__global__ void __launch_bounds__(kPushThreads, kPushCtas) k_push_tiled(const __grid_constant__ LaunchArgs a,
                                                            const __grid_constant__ TileGrid t,
                                                            const __grid_constant__ CUtensorMap phimap,
                                                            const __grid_constant__ CUtensorMap valmap,
                                                            const __grid_constant__ AffineMap aff) {
    extern __shared__ __align__(128) float4 smem4[];
    constexpr int NCOMP = OP == kPushGrad ? 3 : 1;
    constexpr int NPHI = AFF ? 0 : 3;
    constexpr int NW = kPushThreads / 32;
    constexpr bool CELLS = DP == 3 || DP == 4;   // degrees whose taps fill one or two warp instructions
    __shared__ int wrec[NW][8];
    __shared__ int wscan[NW];
    __shared__ __align__(8) unsigned long long bars8[4];
    __shared__ int s_abort;
    const Geometry& g = a.g;
    const long long n1 = g.n1;
    const int G = gridDim.x, T0 = blockIdx.x, nv = t.nv;
    if (T0 >= t.ntiles) return;
    const int ntl = (t.ntiles - T0 + G - 1) / G;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    float* ring = reinterpret_cast<float*>(smem4);
    const int slot_floats = (NPHI + NCOMP) * nv;
    float* accf = ring + t.stages * slot_floats;
    int* acc = reinterpret_cast<int*>(accf);
    const unsigned bars = smem_addr(bars8);
    for (int i = threadIdx.x; i < (t.cap >> 2); i += kPushThreads)
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
        push_ring_fill<NCOMP, TMA, IT, AFF>(ring, slot_floats, t.stages, bars, j, T0 + j * G, j < ntl, a, a.in, t, phimap,
                                            valmap);

    const unsigned acc_base = smem_addr(accf);
    for (int j = 0; j < ntl; ++j) {
        const TileOrigin o = tile_origin(t, T0 + j * G);
        float* slot = ring + (j % t.stages) * slot_floats;
        float* vslot = slot + NPHI * nv;
        if constexpr (TMA) {
            if (!mbar_wait(bars + 8u * (j % t.stages), (unsigned)((j / t.stages) & 1))) s_abort = 1;
        } else {   // this thread's own copies of tile j are done; up to stages - 1 later tiles' still in flight
            wait_groups(t.stages - 1);
        }
        const PushTile pt(o, t, g);
        const PushPos<AFF> pos{slot, nv, &aff};

        // ---- footprint box, sum and maximum of |value| -----------------------
        // bounds of the positions (the first tap is monotone in the position), as keys
        int mn[3], mx[3];
        float ssum = 0.f, smax = 0.f;
        {
            const float inf = __int_as_float(0x7f800000);
            float lo[3] = {inf, inf, inf}, hi[3] = {-inf, -inf, -inf};
            // branch free, so that several voxels' shared loads are in flight
#pragma unroll 4
            for (int lin = threadIdx.x; lin < nv; lin += kPushThreads) {
                float x[3];
                const bool ok = pos(g, pt, lin, x[0], x[1], x[2]) & pt.inside(lin);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    lo[k] = fminf(lo[k], ok ? x[k] : inf);
                    hi[k] = fmaxf(hi[k], ok ? x[k] : -inf);
                }
                bool fin = ok;
                float s1 = 0.f;
#pragma unroll
                for (int p = 0; p < NCOMP; ++p) {
                    const float v = vslot[p * nv + lin];
                    fin = fin & finitef(v);
                    s1 += fabsf(v);
                }
                s1 = fin ? s1 : 0.f;
                ssum += s1;
                smax = fmaxf(smax, s1);
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                mn[k] = float_key(lo[k]);
                mx[k] = float_key(hi[k]);
            }
        }
        auto combine = [&](bool bounds) { tile_combine(wrec, bounds, mn, mx, ssum, smax); };
        combine(true);
        if (s_abort) break;
        PushBox box;
        if (box_place<DP>(mn, mx, g, box)) {
            if constexpr (CELLS) {
                // contracted: the two-word accumulators of a channel group, the
                // sorted voxels, their tags and the cell starts fit the budget
                const long long nce = (long long)(box.e[0] - DP + 1) * (box.e[1] - DP + 1) * (box.e[2] - DP + 1);
                if (nce * kCellMin<DP, OP> <= pt.count(t) && nce < 1024) {
                    long long P = box.e[0] + 3;
                    P += (4 - P) & 7;                 // odd multiples of 4, and planes 16 banks apart:
                    long long Q = P * box.e[1];       // a cell's taps fall in distinct banks
                    Q += (16 - Q) & 31;
                    const long long sz = (Q * box.e[2] + 7) & ~3LL;
                    const long long rows = (kCellBatch + nce + 2) / 2;
                    const long long fixed = kCellBatch + nce + 1;
                    const long long one = 2 * sz + rows * (OP == kPushGrad ? 12 : 8) + fixed;
                    const long long grp = 2 * kCellChannels * sz + rows * 12 + fixed;
                    if (one <= t.cap) {
                        box.cells = (int)nce;
                        box.group = OP == kPush && g.nc > 1 && grp <= t.cap;
                        box.size = (int)sz;
                        box.P = (int)P;
                        box.Q = (int)Q;
                        box.vec = (g.d0[0] & 3) == 0;
                        box.mode = 1;
                    }
                }
            }
            if (!box.cells) box_pitches(t, (t.cap >> 1) & ~3, g, box);
        }
        if (box.mode == 2) {
            for (int lin = threadIdx.x; lin < nv; lin += kPushThreads) {
                float x0, x1, x2;
                if (pt.inside(lin) && pos(g, pt, lin, x0, x1, x2))
                    push_tile_fallback<DP, OP, IT>(a, o.b, (long long)pt.index<IT>(lin), x0, x1, x2);
            }
        } else if (box.mode == 1) {
            const float* inb = a.in + (long long)o.b * g.nc * NCOMP * n1;
            const int bxo = box.lo[0], by0 = box.lo[1], bz0 = box.lo[2];
            auto cell_tile = [&](auto nval_c) {
                constexpr int NVAL = decltype(nval_c)::value;
                constexpr int GRP = OP == kPush ? NVAL : 1;       // channels at once
                const int nce = box.cells, half = box.size;
                const int c0 = box.e[0] - DP + 1, c01 = c0 * (box.e[1] - DP + 1);
                const int rows = (kCellBatch + nce + 2) / 2;
                CellArrays ca;
                ca.A = reinterpret_cast<float4*>(accf + 2 * GRP * half);
                ca.B = ca.A + rows;
                ca.C = ca.B + rows;
                ca.tag = reinterpret_cast<unsigned*>(NVAL > 1 ? ca.C + rows : ca.C);
                ca.start = reinterpret_cast<int*>(ca.tag + kCellBatch);
                for (int cg = 0; cg < g.nc; cg += GRP) {
                    // value p of voxel lin: the ring holds channel 0's
                    auto value = [&](int lin, int p) -> float {
                        const int comp = OP == kPushGrad ? cg * 3 + p : cg + p;
                        if (OP == kPush && cg + p >= g.nc) return 0.f;
                        if (comp < NCOMP) return vslot[comp * nv + lin];
                        return __ldg(inb + (long long)comp * n1 + pt.index<IT>(lin));
                    };
                    // scale of every channel of the group
                    float inv[GRP];
                    int Es[GRP];
                    bool bad = false;
                    float sums[GRP];
                    sums[0] = ssum;
                    if (cg > 0 || GRP > 1) {
                        // one pass over the values of all the group's channels
#pragma unroll
                        for (int q = 0; q < GRP; ++q) sums[q] = 0.f;
#pragma unroll 2
                        for (int lin = threadIdx.x; lin < nv; lin += kPushThreads) {
                            float v[NVAL], x0, x1, x2;
                            const bool in = pt.inside(lin);
#pragma unroll
                            for (int p = 0; p < NVAL; ++p) v[p] = in ? value(lin, p) : 0.f;
                            const bool ok = pos(g, pt, lin, x0, x1, x2) & in;
                            if constexpr (OP == kPushGrad) {
                                const bool fin = ok & finitef(v[0]) & finitef(v[1]) & finitef(v[2]);
                                sums[0] += fin ? fabsf(v[0]) + fabsf(v[1]) + fabsf(v[2]) : 0.f;
                            } else {
#pragma unroll
                                for (int q = 0; q < GRP; ++q) sums[q] += ok & finitef(v[q]) ? fabsf(v[q]) : 0.f;
                            }
                        }
#pragma unroll
                        for (int q = 0; q < GRP; ++q) {
                            ssum = sums[q];
                            __syncthreads();
                            combine(false);
                            sums[q] = ssum;
                        }
                    }
#pragma unroll
                    for (int q = 0; q < GRP; ++q) {
                        Es[q] = scale_exponent(NCOMP == 3 ? 2.f * sums[q] : sums[q]);
                        bad = bad || Es[q] == INT_MIN;
                        if (Es[q] == INT_MIN || Es[q] == INT_MAX) Es[q] = 0;
                        inv[q] = pow2f(22 - Es[q]);
                    }
                    if (bad) return cg;      // non-finite or extreme sums: the caller's float accumulation
                    int base0[GRP];
#pragma unroll
                    for (int q = 0; q < GRP; ++q)
                        base0[q] = box_base(box, g, a.out + ((long long)o.b * g.nc + min(cg + q, g.nc - 1)) * g.n0);
                    for (int l0 = 0; l0 < nv; l0 += kCellBatch) {
                        const int nb = min(kCellBatch, nv - l0);
                        for (int i = threadIdx.x; i <= nce; i += kPushThreads) ca.start[i] = 0;
                        __syncthreads();
                        // count and rank
                        for (int i = threadIdx.x; i < nb; i += kPushThreads) {
                            unsigned tag = ~0u;
                            float x0, x1, x2;
                            if (pt.inside(l0 + i) && pos(g, pt, l0 + i, x0, x1, x2)) {
                                const int cell = (first_tap32(x0, DP) - bxo) + c0 * (first_tap32(x1, DP) - by0) +
                                                 c01 * (first_tap32(x2, DP) - bz0);
                                tag = (unsigned)cell << 16 | (unsigned)atomicAdd(ca.start + cell, 1);
                            }
                            ca.tag[i] = tag;
                        }
                        __syncthreads();
                        // exclusive scan of the counts, rounded up to even
                        {
                            const int per = (nce + kPushThreads - 1) / kPushThreads, i0 = threadIdx.x * per;
                            int cnt[(1024 + kPushThreads - 1) / kPushThreads], sum = 0;
#pragma unroll
                            for (int k = 0; k < (1024 + kPushThreads - 1) / kPushThreads; ++k) {
                                cnt[k] = k < per && i0 + k < nce ? ca.start[i0 + k] : 0;
                                sum += (cnt[k] + 1) & ~1;
                            }
                            int inc = sum;
#pragma unroll
                            for (int d = 1; d < 32; d <<= 1) {
                                const int v = __shfl_up_sync(0xffffffffu, inc, d);
                                if (lane >= d) inc += v;
                            }
                            if (lane == 31) wscan[warp] = inc;
                            __syncthreads();
                            int at = inc - sum;
                            for (int w = 0; w < warp; ++w) at += wscan[w];
#pragma unroll
                            for (int k = 0; k < (1024 + kPushThreads - 1) / kPushThreads; ++k) {
                                if (k < per && i0 + k < nce) {
                                    ca.start[i0 + k] = at;
                                    if (cnt[k] & 1) {       // the odd cell's filler: value 0
                                        const int t2 = (at + cnt[k]) >> 1;
                                        float* A1 = reinterpret_cast<float*>(ca.A + t2);
                                        float* B1 = reinterpret_cast<float*>(ca.B + t2);
                                        A1[1] = A1[3] = B1[1] = B1[3] = 0.f;
                                        if constexpr (NVAL > 1) {
                                            float* C1 = reinterpret_cast<float*>(ca.C + t2);
                                            C1[1] = C1[3] = 0.f;
                                        }
                                    }
                                    at += (cnt[k] + 1) & ~1;
                                }
                            }
                            if (threadIdx.x == kPushThreads - 1) ca.start[nce] = at;
                        }
                        __syncthreads();
                        // place
                        for (int i = threadIdx.x; i < nb; i += kPushThreads) {
                            const unsigned tag = ca.tag[i];
                            if (tag == ~0u) continue;
                            const int at = ca.start[tag >> 16] + (int)(tag & 0xffffu), t2 = at >> 1, u = at & 1;
                            float x[3];
                            pos(g, pt, l0 + i, x[0], x[1], x[2]);
                            float v[3];
                            bool fin = true;
#pragma unroll
                            for (int p = 0; p < NVAL; ++p) {
                                v[p] = value(l0 + i, p);
                                if (OP == kPush) v[p] = finitef(v[p]) ? v[p] : 0.f;
                                else fin = fin & finitef(v[p]);
                            }
                            if (!fin) v[0] = v[1] = v[2] = 0.f;
                            float* A1 = reinterpret_cast<float*>(ca.A + t2) + u;
                            float* B1 = reinterpret_cast<float*>(ca.B + t2) + u;
                            A1[0] = cell_position<DP>(x[0], ceilf(__fsub_rn(x[0], 0.5f * DP)));
                            A1[2] = cell_position<DP>(x[1], ceilf(__fsub_rn(x[1], 0.5f * DP)));
                            B1[0] = cell_position<DP>(x[2], ceilf(__fsub_rn(x[2], 0.5f * DP)));
                            B1[2] = v[0];
                            if constexpr (NVAL > 1) {
                                float* C1 = reinterpret_cast<float*>(ca.C + t2) + u;
                                C1[0] = v[1];
                                C1[2] = v[2];
                            }
                        }
                        __syncthreads();
                        // channels of a group start at their own alignment: their base offsets differ
                        cell_scatter<DP, OP, NVAL>(ca, nce, c0, c01, acc_base, box.P, box.Q, half, inv, base0);
                        __syncthreads();
                    }
#pragma unroll
                    for (int q = 0; q < GRP; ++q) {
                        if (cg + q >= g.nc) break;
                        int b0, b1, b2;
                        bnd_code(a, cg + q, b0, b1, b2);
                        FixedScale fs;
                        fs.set(Es[q], 43);
                        int* hi = acc + 2 * q * half;
                        push_flush<IT>(box, g, b0, b1, b2, a.out + ((long long)o.b * g.nc + cg + q) * g.n0, base0[q],
                                       [&](int w) {
                                           const int4 h = *reinterpret_cast<const int4*>(hi + w);
                                           const int4 l = *reinterpret_cast<const int4*>(hi + half + w);
                                           *reinterpret_cast<int4*>(hi + w) = make_int4(0, 0, 0, 0);
                                           *reinterpret_cast<int4*>(hi + half + w) = make_int4(0, 0, 0, 0);
                                           return make_float4(fixed_value(h.x, l.x, fs), fixed_value(h.y, l.y, fs),
                                                              fixed_value(h.z, l.z, fs), fixed_value(h.w, l.w, fs));
                                       },
                                       [&](int w) {
                                           const int h = hi[w], l = hi[half + w];
                                           hi[w] = 0;
                                           hi[half + w] = 0;
                                           return fixed_value(h, l, fs);
                                       });
                    }
                    __syncthreads();
                }
                return g.nc;
            };
            int first = 0;
            if constexpr (CELLS) {
                if (box.cells > 0) {
                    if constexpr (OP == kPushGrad) first = cell_tile(std::integral_constant<int, 3>{});
                    else first = box.group ? cell_tile(std::integral_constant<int, kCellChannels>{})
                                          : cell_tile(std::integral_constant<int, 1>{});
                    // the sorted voxels sat in the accumulator's words: clear them
                    for (int i = threadIdx.x; i < (t.cap >> 2); i += kPushThreads)
                        reinterpret_cast<float4*>(accf)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (first < g.nc) {
                        __syncthreads();
                        ssum = smax = 0.f;
                    }
                }
            }
            for (int c = first; c < g.nc; ++c) {
                int b0, b1, b2;
                bnd_code(a, c, b0, b1, b2);
                if (c > 0 || box.cells > 0) {
                    // values of channel c over channel 0's in this thread's ring words
                    ssum = smax = 0.f;
#pragma unroll 2
                    for (int lin = threadIdx.x; lin < nv; lin += kPushThreads) {
                        if (!pt.inside(lin)) continue;
                        const IT v = pt.index<IT>(lin);
                        bool fin = true;
                        float s1 = 0.f;
#pragma unroll
                        for (int p = 0; p < NCOMP; ++p) {
                            const float vv = __ldg(inb + (long long)c * NCOMP * n1 + v + p * n1);   // (c = 0: again)
                            vslot[p * nv + lin] = vv;
                            fin = fin && finitef(vv);
                            s1 += fabsf(vv);
                        }
                        float x0, x1, x2;
                        if (!fin || !pos(g, pt, lin, x0, x1, x2)) continue;
                        ssum += s1;
                        smax = fmaxf(smax, s1);
                    }
                    __syncthreads();   // the previous channel's flush and record reads are done
                    combine(false);
                }
                push_channel<DP, OP, IT>(g, t, pt, pos, vslot, box, b0, b1, b2,
                                         a.out + ((long long)o.b * g.nc + c) * g.n0, accf, ssum, smax);
            }
        }
        if (TMA && g.nc > 1) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();   // ring slot j is free and the accumulator is clear
        push_ring_fill<NCOMP, TMA, IT, AFF>(ring, slot_floats, t.stages, bars, j + t.stages, T0 + (j + t.stages) * G,
                                            j + t.stages < ntl, a, a.in, t, phimap, valmap);
    }
    if constexpr (!TMA) asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// Tile grid of a push launch: ring depth for the shared memory that kPushCtas resident
// CTAs per SM leave; one slot, and fewer CTAs, for budgets too large for that.
TileGrid push_grid(const LaunchArgs& a, const TileCfg& c, int comps, size_t& smem) {
    TileGrid t = make_grid(a, c);
    t.nv = 1 << (c.lx + c.ly + c.lz);
    t.pmod = (1 << c.lx) & 31;
    const size_t slot = (size_t)comps * t.nv * 4, accb = (size_t)c.cap * 4;
    t.stages = 4;
    while (t.stages > 1 && t.stages * slot + accb > (226 / kPushCtas - 1) * 1024) --t.stages;
    smem = t.stages * slot + accb;
    return t;
}

template <int DP, int OP, typename IT, bool AFF>
cudaError_t launch_push_one(const LaunchArgs& a, const TileCfg& c, cudaStream_t s, const AffineMap& aff) {
    constexpr int NCOMP = OP == kPushGrad ? 3 : 1;
    CUtensorMap phimap, valmap;
    std::memset(&phimap, 0, sizeof phimap);
    std::memset(&valmap, 0, sizeof valmap);
    size_t smem;
    const TileGrid t = push_grid(a, c, NCOMP + (AFF ? 0 : 3), smem);
    const bool tma = (AFF || encode_tile_map(&phimap, a.phi, a.g.d1, 3LL * a.g.nb, t, 3)) &&
                     encode_tile_map(&valmap, a.in, a.g.d1, (long long)NCOMP * a.g.nc * a.g.nb, t, NCOMP);
    if (tma) return launch_persistent(k_push_tiled<DP, OP, IT, true, AFF>, t, smem, s, kPushThreads, a, t, phimap, valmap, aff);
    return launch_persistent(k_push_tiled<DP, OP, IT, false, AFF>, t, smem, s, kPushThreads, a, t, phimap, valmap, aff);
}

template <int OP, typename IT, bool AFF = false>
cudaError_t push_dispatch(const LaunchArgs& a, const TileCfg& t, cudaStream_t s, const AffineMap& aff = AffineMap{}) {
    switch (a.g.dp[0]) {
        case 1: return launch_push_one<1, OP, IT, AFF>(a, t, s, aff);
        case 2: return launch_push_one<2, OP, IT, AFF>(a, t, s, aff);
        case 3: return launch_push_one<3, OP, IT, AFF>(a, t, s, aff);
        case 4: return launch_push_one<4, OP, IT, AFF>(a, t, s, aff);
        default: return launch_push_one<5, OP, IT, AFF>(a, t, s, aff);
    }
}

}  // namespace
}  // namespace pp
