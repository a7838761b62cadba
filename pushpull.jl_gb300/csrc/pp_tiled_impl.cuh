// pp_tiled_impl.cuh -- shared-memory tiled pull family and privatised push family.
//
// Included by the pp_tiled*.cu translation units, each of which instantiates
// one group of kernels (so the library compiles in parallel); everything here
// has internal linkage, the device status word included (one per unit, read
// and combined by read_device_status).
//
// A CTA owns a TX x TY x TZ tile of sample voxels (power-of-two sides, up to
// 256*V voxels for 256 threads).  It reads the tile's deformation once,
// reduces the integer first taps to the tile's footprint box in the image
//   [min o, max o + dp - 1]  per dimension,
// and, when the box fits its shared-memory budget:
//   pull:  stages the box once per channel -- boundary folding and the DST-II
//          sign are applied while staging, so taps index the box directly with
//          no per-tap modulo -- then evaluates every voxel from shared memory;
//   push:  zeroes a box-sized accumulator, scatters every voxel's weighted taps
//          into it with shared-memory atomics, then flushes the box to the
//          image with one global reduction per non-zero element (4-wide vector
//          reductions on aligned interior runs) instead of dp^3 global atomics
//          per voxel.
// Tiles whose footprint does not fit (large local expansion, far-out
// coordinates) take the per-voxel global path for that tile only.
//
// Latency: each CTA is persistent and walks a sequence of tiles.  The
// deformation of the next kStages tiles (and, for push, their channel-0 values)
// streams into a ring of shared-memory slots with TMA bulk tensor copies that
// complete on mbarriers, so several tiles' worth of HBM reads are in flight per
// SM while the current tile computes.  Pull additionally stages the next tile's
// image box with cp.async into a second buffer.
//
// Bank layout: lanes of a warp cover TX consecutive x of the tile and
// 32/TX consecutive tile rows in y.  The box row pitch P is chosen with
// P % 32 == TX % 32, so for a smooth deformation the rows of one warp land in
// disjoint bank ranges (TX = 32: bank = x mod 32 in every row).
//
// Reference kernels replaced: pull_element / pullg_element / pullh_element /
// push_element / pushg_element (artifacts/C/pushpull.cu:33-163); per-voxel math
// pull1 / pullg1 / pullh1 / push1 / pushg1 (artifacts/C/pushpull_dev.cu:61-179).
#include <climits>
#include <cstring>
#include <map>
#include <mutex>
#include <utility>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "pp_tiled.cuh"
#include "pp_voxel.cuh"

namespace pp {
namespace {

// Device status word of this translation unit: bits record bounded waits that
// gave up (read and cleared through read_device_status).
__device__ unsigned int g_device_status;

unsigned unit_status(bool reset) {
    unsigned v = 0;
    if (cudaMemcpyFromSymbol(&v, g_device_status, sizeof v) != cudaSuccess) return 0xffffffffu;
    if (reset) {
        const unsigned z = 0;
        cudaMemcpyToSymbol(g_device_status, &z, sizeof z);
    }
    return v;
}

constexpr int kThreads = 256;
constexpr int kStages = 4;                 // tiles of the ring in flight per CTA
constexpr unsigned kStatusWaitTimeout = 1u;
constexpr int kClamp = 1 << 29;    // first taps are clamped to +-kClamp for the box reduction
// Fixed image window for TMA-staged pull boxes: row pitch 24 (24 % 32 places
// the 4 rows of an 8-wide warp tile in disjoint bank ranges), 16 rows, 16 planes.
constexpr int kTmaBoxX = 24, kTmaBoxY = 16, kTmaBoxZ = 16;
constexpr int kTmaBoxFloats = kTmaBoxX * kTmaBoxY * kTmaBoxZ;

template <int DP, int ORD>
struct W3 {
    float w[DP];
    float dw[ORD >= 1 ? DP : 1];
    float hw[ORD >= 2 ? DP : 1];
};

// One spline row of DP consecutive box elements, addressed with immediate
// offsets from one shared-memory base address (one asm statement per row).
template <int DP>
__device__ __forceinline__ void lds_row(unsigned a, float (&f)[DP]) {
    if constexpr (DP == 1) {
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(f[0]) : "r"(a));
    } else if constexpr (DP == 2) {
        asm volatile("ld.shared.f32 %0, [%2];\n\tld.shared.f32 %1, [%2+4];" : "=f"(f[0]), "=f"(f[1]) : "r"(a));
    } else if constexpr (DP == 3) {
        asm volatile("ld.shared.f32 %0, [%3];\n\tld.shared.f32 %1, [%3+4];\n\tld.shared.f32 %2, [%3+8];"
                     : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]) : "r"(a));
    } else if constexpr (DP == 4) {
        asm volatile("ld.shared.f32 %0, [%4];\n\tld.shared.f32 %1, [%4+4];\n\tld.shared.f32 %2, [%4+8];\n\t"
                     "ld.shared.f32 %3, [%4+12];"
                     : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]) : "r"(a));
    } else {
        asm volatile("ld.shared.f32 %0, [%5];\n\tld.shared.f32 %1, [%5+4];\n\tld.shared.f32 %2, [%5+8];\n\t"
                     "ld.shared.f32 %3, [%5+12];\n\tld.shared.f32 %4, [%5+16];"
                     : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]), "=f"(f[4]) : "r"(a));
    }
}

// Integer reductions of DP consecutive box words (one asm statement per row).
template <int DP>
__device__ __forceinline__ void red_row_s32(unsigned a, const int (&v)[DP]) {
    if constexpr (DP == 1) {
        asm volatile("red.shared.add.s32 [%0], %1;" ::"r"(a), "r"(v[0]) : "memory");
    } else if constexpr (DP == 2) {
        asm volatile("red.shared.add.s32 [%0], %1;\n\tred.shared.add.s32 [%0+4], %2;" ::"r"(a), "r"(v[0]), "r"(v[1])
                     : "memory");
    } else if constexpr (DP == 3) {
        asm volatile("red.shared.add.s32 [%0], %1;\n\tred.shared.add.s32 [%0+4], %2;\n\t"
                     "red.shared.add.s32 [%0+8], %3;" ::"r"(a), "r"(v[0]), "r"(v[1]), "r"(v[2])
                     : "memory");
    } else if constexpr (DP == 4) {
        asm volatile("red.shared.add.s32 [%0], %1;\n\tred.shared.add.s32 [%0+4], %2;\n\t"
                     "red.shared.add.s32 [%0+8], %3;\n\tred.shared.add.s32 [%0+12], %4;" ::"r"(a), "r"(v[0]),
                     "r"(v[1]), "r"(v[2]), "r"(v[3])
                     : "memory");
    } else {
        asm volatile("red.shared.add.s32 [%0], %1;\n\tred.shared.add.s32 [%0+4], %2;\n\t"
                     "red.shared.add.s32 [%0+8], %3;\n\tred.shared.add.s32 [%0+12], %4;\n\t"
                     "red.shared.add.s32 [%0+16], %5;" ::"r"(a), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4])
                     : "memory");
    }
}

struct Box {
    int lo[3];      // minima of the first taps
    int xo;         // x origin of the box in shared memory: lo[0] rounded down to a multiple of 4
    int ext[3];     // box extent (x counted from xo)
    int P, Q, size; // row pitch (P % 32 == pmod, P % 4 == 0), plane pitch (multiple of 32), floats
    int mode;       // 0 no valid voxel, 1 shared memory, 2 per-voxel global fallback
    int base;       // warp-specialised pull: first word of the box in its buffer (0..3)
    int interior;   // bit k: the box lies inside the image along dimension k (no folding)
    int tma;        // 1: the box is a fixed window loaded by one TMA copy; 2: the same, with mirrored margins to
                    // complete; 3: loaded row by row; 4: the same, DST-II signs to apply
    float S;        // block sum of the caller's per-thread value (push: bound on sum |contribution|)
    int E;          // scale exponent of the fixed-point accumulator for S (see scale_exponent)
};

// Exponent E of the fixed-point accumulator scale for a bound S on the sum of
// |contributions|: S < 2^E.  INT_MAX: nothing to accumulate (S == 0);
// INT_MIN: S non-finite or outside the range the scale factors cover, so the
// tile accumulates in float instead.
__device__ __forceinline__ int scale_exponent(float S) {
    if (S == 0.f) return INT_MAX;
    if (!(S > 0.f) || !finitef(S)) return INT_MIN;
    int E;
    frexpf(S * 1.0009765625f, &E);
    return (E < -80 || E > 100) ? INT_MIN : E;
}

// Block-wide reduction of the first-tap bounds into the footprint box.
// `words` = shared-memory words needed per box element (1 for pull, 2 for push).
// Also sums `ssum` over the block into box.S (fixed order) and sets box.E.
template <int DP>
__device__ __forceinline__ void reduce_box(int (&mn)[3], int (&mx)[3], const TileGrid& t, const Geometry& g,
                                           int words, Box& box, int (&red)[8][7], float ssum = 0.f) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        mn[k] = __reduce_min_sync(0xffffffffu, mn[k]);
        mx[k] = __reduce_max_sync(0xffffffffu, mx[k]);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ssum += __shfl_xor_sync(0xffffffffu, ssum, off);
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            red[warp][k] = mn[k];
            red[warp][3 + k] = mx[k];
        }
        red[warp][6] = __float_as_int(ssum);
    }
    __syncthreads();
    if (warp == 0) {
        // warp 0 combines the per-warp records (lane w < 8 holds warp w's)
        constexpr int NW = kThreads / 32;
        int lo[3], hi[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lo[k] = __reduce_min_sync(0xffffffffu, lane < NW ? red[lane][k] : INT_MAX);
            hi[k] = __reduce_max_sync(0xffffffffu, lane < NW ? red[lane][3 + k] : INT_MIN);
        }
        // the scale bound is summed in a fixed order (warp 0, 1, ...): lane 0 alone
        float S = 0.f;
        if (lane == 0)
            for (int w = 0; w < NW; ++w) S += __int_as_float(red[w][6]);
        if (lane == 0) {
        box.S = S;
        box.E = scale_exponent(S);
        if (lo[0] > hi[0]) {
            box.mode = 0;
            box.tma = 0;
        } else {
            const int xo = lo[0] & ~3;
            long long e[3];
            e[0] = (long long)hi[0] + DP - xo;
            e[1] = (long long)hi[1] + DP - lo[1];
            e[2] = (long long)hi[2] + DP - lo[2];
            int interior = 0;
            if (xo >= 0 && (long long)hi[0] + DP <= g.d0[0]) interior |= 1;
            if (lo[1] >= 0 && (long long)hi[1] + DP <= g.d0[1]) interior |= 2;
            if (lo[2] >= 0 && (long long)hi[2] + DP <= g.d0[2]) interior |= 4;
            // P % 32 == pmod and Q % 32 == 0 keep the warp's rows and planes in
            // disjoint banks; when that padding would not fit, pack tightly.
            long long P = 0, Q = 0;
            P = (e[0] + 3) & ~3LL;
            long long Pp = P + (((t.pmod - (int)(P & 31)) + 32) & 31);
            Q = (Pp * e[1] + 31) & ~31LL;
            if (Q * e[2] * words <= t.cap) {
                P = Pp;
            } else {
                Q = (P * e[1] + 3) & ~3LL;
            }
            long long size = Q * e[2];
            const bool fits = e[0] <= 4096 && e[1] <= 4096 && e[2] <= 4096 && size * words <= t.cap;
            box.mode = fits ? 1 : 2;
            box.tma = 0;
            if (words == 1 && t.img_tma && interior == 7 && e[0] <= kTmaBoxX && e[1] <= kTmaBoxY &&
                e[2] <= kTmaBoxZ) {
                box.mode = 1;
                box.tma = 1;
                P = kTmaBoxX;
                Q = kTmaBoxX * kTmaBoxY;
                size = kTmaBoxFloats;
            }
            const bool staged = box.mode == 1;
            box.lo[0] = lo[0];
            box.lo[1] = lo[1];
            box.lo[2] = lo[2];
            box.xo = xo;
#pragma unroll
            for (int k = 0; k < 3; ++k) box.ext[k] = staged ? (int)e[k] : 0;
            box.P = staged ? (int)P : 0;
            box.Q = staged ? (int)Q : 0;
            box.size = staged ? (int)size : 0;
            box.interior = interior;
        }
        }
    }
    __syncthreads();
}

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem_src) : "memory");
}

__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gmem_src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(gmem_src) : "memory");
}

// Rows of the box are distributed over warps; within a warp a group of `lpr`
// lanes (a power of two) shares a row.
template <int NT = kThreads>
struct RowWalk {
    int lg, sub, e0;   // lanes per row = 1 << lg
    int ry, rz;        // this lane group's current row
    int sy, sz;        // row step split into (y, z) parts
    int ey;
    __device__ __forceinline__ RowWalk(int items_per_row, int ey_) {
        const int n = items_per_row < 1 ? 1 : (items_per_row > 32 ? 32 : items_per_row);
        lg = 32 - __clz(n - 1);                       // ceil(log2 n)
        const int lane = threadIdx.x & 31;
        sub = lane >> lg;
        e0 = lane & ((1 << lg) - 1);
        ey = ey_;
        const int first = (threadIdx.x >> 5) * (32 >> lg) + sub;
        const int step = (NT / 32) * (32 >> lg);
        rz = first / ey;
        ry = first - rz * ey;
        sz = step / ey;
        sy = step - sz * ey;
    }
    __device__ __forceinline__ int lpr() const { return 1 << lg; }
    __device__ __forceinline__ void next() {
        ry += sy;
        rz += sz;
        if (ry >= ey) {
            ry -= ey;
            ++rz;
        }
    }
};

// Folded walk over the box: fn(sm_index, global_index, sign) once per element.
template <typename IT, class FN>
__device__ __forceinline__ void walk_box(const Box& box, const Geometry& g, int b0, int b1, int b2, FN fn) {
    const int ex = box.ext[0], ey = box.ext[1], ez = box.ext[2];
    RowWalk<> rw(ex, ey);
    const IT sy = (IT)g.d0[0];
    const IT sz = (IT)(g.d0[0] * g.d0[1]);
    const bool xin = box.interior & 1, yin = box.interior & 2, zin = box.interior & 4;
    for (; rw.rz < ez; rw.next()) {
        const int rz = rw.rz, ry = rw.ry;
        float sgy = 1.f, sgz = 1.f;
        const IT gy = yin ? (IT)(box.lo[1] + ry) : (IT)fold_tap(b1, (long long)box.lo[1] + ry, g.d0[1], sgy);
        const IT gz = zin ? (IT)(box.lo[2] + rz) : (IT)fold_tap(b2, (long long)box.lo[2] + rz, g.d0[2], sgz);
        const IT rowg = gz * sz + gy * sy;
        const int rsm = rz * box.Q + ry * box.P;
        const float syz = sgy * sgz;
        if (xin) {
            const IT base = rowg + (IT)box.xo;
            for (int e = rw.e0; e < ex; e += rw.lpr()) fn(rsm + e, base + (IT)e, syz);
        } else {
            for (int e = rw.e0; e < ex; e += rw.lpr()) {
                float sgx;
                const IT gx = (IT)fold_tap(b0, (long long)box.xo + e, g.d0[0], sgx);
                fn(rsm + e, rowg + gx, syz * sgx);
            }
        }
    }
}

// Stage one channel of the image box into shared memory without waiting: the
// caller commits the cp.async group and waits for it before the box is read
// (the pull kernels overlap the next tile's staging with this tile's work).
// Interior boxes of a 16-byte aligned image with d0[0] % 4 == 0 copy whole
// 16-byte row chunks; other boxes fold (and sign) per element.
template <typename IT>
__device__ __forceinline__ void stage_box(const Box& box, const Geometry& g, int b0, int b1, int b2,
                                          const float* f0, float* sm) {
    if (box.interior == 7 && (g.d0[0] & 3) == 0 && (reinterpret_cast<uintptr_t>(f0) & 15) == 0) {
        const int ey = box.ext[1], ez = box.ext[2];
        const int n4 = (box.ext[0] + 3) >> 2;
        RowWalk<> rw(n4, ey);
        const IT sy = (IT)g.d0[0];
        const IT sz = (IT)(g.d0[0] * g.d0[1]);
        for (; rw.rz < ez; rw.next()) {
            const int rz = rw.rz, ry = rw.ry;
            const float* src = f0 + ((IT)(box.lo[2] + rz) * sz + (IT)(box.lo[1] + ry) * sy + (IT)box.xo);
            float* dst = sm + (rz * box.Q + ry * box.P);
            for (int ch = rw.e0; ch < n4; ch += rw.lpr()) cp_async16(dst + 4 * ch, src + 4 * ch);
        }
        return;
    }
    // folded boxes: elements with sign +1 are copied asynchronously as well;
    // mirrored DST-II elements (sign -1 or 0) are loaded and signed here
    walk_box<IT>(box, g, b0, b1, b2, [&](int si, IT gi, float s) {
        if (s == 1.f) cp_async4(sm + si, f0 + gi);
        else sm[si] = s * __ldg(f0 + gi);
    });
}

// A footprint box as row loaders see it: origin in the image, extents, pitches, first
// word, and whether rows fold (in y or z).
struct RowBox {
    int lo[3], e[3], P, Q, base;
    bool fold;
};

// NT threads load one channel of a box row by row with cp.async, eight lanes to a
// row, folding rows and elements outside the image onto their sources (no signs:
// see sign_rows).  The caller commits and waits.  Rows that have the same 16-byte
// alignment in the image and in the box copy whole chunks (three words lie between
// rows: a row's first and last chunk may overwrite them); chunks at the image's x
// ends, and rows whose alignment differs, copy elements.
template <int NT, typename IT>
__device__ __forceinline__ void load_rows(const RowBox& box, const Geometry& g, int b0, int b1, int b2, const float* f0,
                                          float* sm, int tid) {
    const int ex = box.e[0], ey = box.e[1], rows = ey * box.e[2], dx = (int)g.d0[0];
    const IT sy = (IT)g.d0[0];
    const IT sz = (IT)(g.d0[0] * g.d0[1]);
    constexpr int RS = NT / 8;   // rows at a time
    const int sub = tid >> 3, l8 = tid & 7;
    int rz = sub / ey, ry = sub - rz * ey;
    const int sz_step = RS / ey, sy_step = RS - sz_step * ey;
    const int fw = (int)((reinterpret_cast<uintptr_t>(f0) >> 2) & 3) + box.lo[0];
    for (int r = sub; r < rows; r += RS) {
        IT gy = (IT)(box.lo[1] + ry), gz = (IT)(box.lo[2] + rz);
        if (box.fold) {
            float s;
            gy = (IT)fold_tap(b1, (long long)box.lo[1] + ry, g.d0[1], s);
            gz = (IT)fold_tap(b2, (long long)box.lo[2] + rz, g.d0[2], s);
        }
        const IT ro = gz * sz + gy * sy;
        const float* grow = f0 + ro;
        const int si = box.base + rz * box.Q + ry * box.P;
        const int mis = (fw + (int)(ro & 3)) & 3;
        const bool same = (si & 3) == mis;
        for (int e = 4 * l8 - mis; e < ex; e += 32) {
            const int gx = box.lo[0] + e;
            if (same && gx >= 0 && gx + 4 <= dx) {
                cp_async16(sm + si + e, grow + gx);
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (e + u < 0 || e + u >= ex) continue;
                    float s;
                    const IT fx = (IT)fold_tap(b0, (long long)gx + u, g.d0[0], s);
                    cp_async4(sm + si + e + u, grow + fx);
                }
            }
        }
        ry += sy_step;
        rz += sz_step;
        if (ry >= ey) {
            ry -= ey;
            ++rz;
        }
    }
}

// DST-II signs of a box loaded by load_rows (all NT threads; the caller
// synchronises them before and afterwards).
template <int NT>
__device__ __forceinline__ void sign_rows(const RowBox& box, const Geometry& g, int b0, int b1, int b2, float* sm,
                                          int tid) {
    const int ex = box.e[0], ey = box.e[1], rows = ey * box.e[2];
    const int lane16 = tid & 15;
    for (int r = tid >> 4; r < rows; r += NT >> 4) {
        const int rz = r / ey, ry = r - rz * ey;
        float s1, s2;
        (void)fold_tap(b1, (long long)box.lo[1] + ry, g.d0[1], s1);
        (void)fold_tap(b2, (long long)box.lo[2] + rz, g.d0[2], s2);
        float* row = sm + box.base + rz * box.Q + ry * box.P;
        for (int e = lane16; e < ex; e += 16) {
            float s0;
            (void)fold_tap(b0, (long long)box.lo[0] + e, g.d0[0], s0);
            if (s0 * s1 * s2 < 0.f) row[e] = -row[e];
        }
    }
}

// ---- push accumulation -----------------------------------------------------
// Each box element holds two int32 words (hi, lo) of a fixed-point sum.  With
// S >= the sum of |contribution| over the tile's channel (B-spline weights are
// non-negative and sum to one per axis; derivative weights sum to at most 2 in
// absolute value) and S < 2^E, a contribution c is split as
//     c = hi * q1 + lo * q2 + rounding,  q1 = 2^(E-22), q2 = 2^(E-43),
// |hi| <= 2^22 and |lo| <= 2^20, so 512 contributions per element cannot
// overflow and the rounding error per element is at most 2^(E-35), i.e.
// below 3e-11 of S.  Both words use native integer shared atomics.  Where E
// is out of range (S = 0, non-finite, or extreme) the tile uses float atomics.
constexpr float kMagic = 12582912.0f;     // 1.5 * 2^23: float -> nearest int for |y| <= 2^22
constexpr int kMagicBits = 0x4B400000;
constexpr float kLoScale = 2097152.0f;    // 2^21 lower quanta per upper one (tiles of up to 1024 voxels)

__device__ __forceinline__ float pow2f(int k) { return __int_as_float((127 + k) << 23); }   // -126 <= k <= 127

struct FixedScale {
    float inv_q1, q1, q2;
    __device__ __forceinline__ void set(int E, int bits = 43) {
        inv_q1 = pow2f(22 - E);
        q1 = pow2f(E - 22);
        q2 = pow2f(E - bits);
    }
};

__device__ __forceinline__ float fixed_value(int h, int l, const FixedScale& fs) {
    return fmaf(__int2float_rn(h), fs.q1, __int2float_rn(l) * fs.q2);
}

// Flush one channel's accumulator box into the image with global reductions:
// interior rows of an aligned image use 4-wide vector reductions on aligned
// groups, all-zero groups are skipped.  `val(si)` reads box element si.
template <typename IT, class VAL>
__device__ __forceinline__ void flush_box(const Box& box, const Geometry& g, int b0, int b1, int b2, float* f0,
                                          VAL val) {
    if ((box.interior & 1) && (g.d0[0] & 3) == 0 && (reinterpret_cast<uintptr_t>(f0) & 15) == 0) {
        const int ey = box.ext[1], ez = box.ext[2];
        const int n4 = (box.ext[0] + 3) >> 2;        // rows start at xo (16-byte aligned); whole groups
        RowWalk<> rw(n4, ey);
        const IT sy = (IT)g.d0[0];
        const IT sz = (IT)(g.d0[0] * g.d0[1]);
        for (; rw.rz < ez; rw.next()) {
            const int rz = rw.rz, ry = rw.ry;
            float sgy = 1.f, sgz = 1.f;
            const IT gy = (box.interior & 2) ? (IT)(box.lo[1] + ry)
                                             : (IT)fold_tap(b1, (long long)box.lo[1] + ry, g.d0[1], sgy);
            const IT gz = (box.interior & 4) ? (IT)(box.lo[2] + rz)
                                             : (IT)fold_tap(b2, (long long)box.lo[2] + rz, g.d0[2], sgz);
            const float s = sgy * sgz;
            float* grow = f0 + (gz * sz + gy * sy + (IT)box.xo);
            const int rsm = rz * box.Q + ry * box.P;
            for (int ch = rw.e0; ch < n4; ch += rw.lpr()) {
                const int e = 4 * ch;
                // elements past the box row (e >= ext) are zero in the accumulator
                const float4 v = make_float4(s * val(rsm + e), s * val(rsm + e + 1), s * val(rsm + e + 2),
                                             s * val(rsm + e + 3));
                if (v.x != 0.f || v.y != 0.f || v.z != 0.f || v.w != 0.f)
                    atomicAdd(reinterpret_cast<float4*>(grow + e), v);
            }
        }
        return;
    }
    walk_box<IT>(box, g, b0, b1, b2, [&](int si, IT gi, float s) {
        const float v = val(si);
        if (v != 0.f) atomicAdd(f0 + gi, s * v);
    });
}

// ---- tiles -----------------------------------------------------------------
struct TileOrigin {
    int b;            // batch
    int x0, y0, z0;   // first sample voxel of the tile
};

// linear tile index (x fastest, batch slowest) -> tile origin
__device__ __forceinline__ TileOrigin tile_origin(const TileGrid& t, int T) {
    const unsigned u = (unsigned)T;
    const unsigned q1 = (unsigned)(((unsigned long long)u * t.mx) >> t.sx);
    const unsigned q2 = (unsigned)(((unsigned long long)q1 * t.my) >> t.sy);
    const unsigned q3 = (unsigned)(((unsigned long long)q2 * t.mz) >> t.sz);
    TileOrigin r;
    r.x0 = (int)(u - q1 * (unsigned)t.ntx) << t.lx;
    r.y0 = (int)(q1 - q2 * (unsigned)t.nty) << t.ly;
    r.z0 = (int)(q2 - q3 * (unsigned)t.ntz) << t.lz;
    r.b = (int)q3;
    return r;
}

// This thread's tile-local voxel coordinates (fixed for the kernel's lifetime)
// and the sample-grid dimensions as 32-bit integers.
template <int V>
struct ThreadVox {
    int vx[V], vy[V], vz[V];
    int D0, D1, D2;
    __device__ __forceinline__ ThreadVox(const TileGrid& t, const Geometry& g) {
#pragma unroll
        for (int q = 0; q < V; ++q) {
            const int lin = threadIdx.x + q * kThreads;
            vx[q] = lin & ((1 << t.lx) - 1);
            vy[q] = (lin >> t.lx) & ((1 << t.ly) - 1);
            vz[q] = lin >> (t.lx + t.ly);
        }
        D0 = (int)g.d1[0];
        D1 = (int)g.d1[1];
        D2 = (int)g.d1[2];
    }
    // index() for a runtime slot lin = threadIdx.x + q * kThreads (no register arrays)
    template <typename IT>
    __device__ __forceinline__ IT index_lin(const TileOrigin& o, int lin, const TileGrid& t) const {
        const int gx = o.x0 + (lin & ((1 << t.lx) - 1));
        const int gy = o.y0 + ((lin >> t.lx) & ((1 << t.ly) - 1));
        const int gz = o.z0 + (lin >> (t.lx + t.ly));
        if (gx >= D0 || gy >= D1 || gz >= D2) return (IT)-1;
        return (IT)gx + (IT)D0 * ((IT)gy + (IT)D1 * (IT)gz);
    }
    // linear sample index of voxel q within its batch, or -1 outside the grid
    template <typename IT>
    __device__ __forceinline__ IT index(const TileOrigin& o, int q) const {
        const int gx = o.x0 + vx[q], gy = o.y0 + vy[q], gz = o.z0 + vz[q];
        if (gx >= D0 || gy >= D1 || gz >= D2) return (IT)-1;
        return (IT)gx + (IT)D0 * ((IT)gy + (IT)D1 * (IT)gz);
    }
};

template <int DP, int OP, typename IT>
__device__ __noinline__ void push_tile_fallback(const LaunchArgs& a, int b, long long v, float x0, float x1,
                                                float x2) {
    push_voxel_global<DP, OP, IT>(a, b, v, x0, x1, x2);
}

// ---- tile ring: per-tile deformation several tiles ahead ----
//
// Slot k of the ring holds one tile laid out as [component][z][y][x] -- exactly
// the order of a 4-D TMA box (TX, TY, TZ, C) -- so the thread owning tile-local
// voxel `lin` reads component k at slot + k*NV + lin.  With TMA, thread 0 fills
// a slot with one bulk tensor copy per tensor that completes on the slot's
// mbarrier; without it (unaligned geometry) the threads fill it with plain loads.

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: gives up after `limit` clock cycles, records the failure in
// the device status word and returns false.  A kernel whose wait gave up skips
// its remaining work and returns; copies it had already issued may still land
// in its shared memory, so after a recorded timeout the context is suspect and
// the caller should treat its outputs as undefined.
constexpr long long kWaitCycles = 4000000000LL;   // about two seconds
__device__ __forceinline__ bool mbar_wait_limit(unsigned bar, unsigned parity, long long limit) {
    if (mbar_try(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try(bar, parity)) {
        if (clock64() - t0 > limit) {
            atomicOr(&g_device_status, kStatusWaitTimeout);
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity) {
    return mbar_wait_limit(bar, parity, kWaitCycles);
}
__device__ __forceinline__ void tma_load_4d(unsigned dst, const CUtensorMap* map, unsigned bar, int x, int y, int z,
                                            int w) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
        "%5}], [%6];" ::"r"(dst),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar)
        : "memory");
}

struct Ring {
    float* base;       // first slot
    int slot_floats;   // floats per slot
    unsigned bars;     // shared address of the first mbarrier
};

// Fill ring slot (j % kStages) with the deformation of tile T.  Called by every thread.
template <int V, bool TMA, typename IT>
__device__ __forceinline__ void ring_fill(const Ring& r, int j, int T, const LaunchArgs& a, const TileGrid& t,
                                          const ThreadVox<V>& tv, const CUtensorMap& phimap) {
    constexpr int NV = kThreads * V;
    float* slot = r.base + (j % kStages) * r.slot_floats;
    const TileOrigin o = tile_origin(t, T);
    if constexpr (TMA) {
        if (threadIdx.x == 0) {
            const unsigned bar = r.bars + 8u * (j % kStages);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_expect_tx(bar, (unsigned)(3 * NV * sizeof(float)));
            tma_load_4d(smem_addr(slot), &phimap, bar, o.x0, o.y0, o.z0, 3 * o.b);
        }
    } else {
        const long long n1 = a.g.n1;
        const float* phi = a.phi + (long long)o.b * 3 * n1;
#pragma unroll
        for (int q = 0; q < V; ++q) {
            const int lin = threadIdx.x + q * kThreads;
            const IT v = tv.template index<IT>(o, q);
#pragma unroll
            for (int k = 0; k < 3; ++k) slot[k * NV + lin] = v < 0 ? 0.f : __ldg(phi + v + k * n1);
        }
    }
}

template <bool TMA>
__device__ __forceinline__ bool ring_wait(const Ring& r, int j) {
    if constexpr (TMA) return mbar_wait(r.bars + 8u * (j % kStages), (unsigned)((j / kStages) & 1));
    return true;
}

// First-tap bounds of this thread's valid voxels of the tile whose deformation is in
// `slot`.
template <int DP, int V, typename IT>
__device__ __forceinline__ void tile_bounds(const Geometry& g, const TileOrigin& o, const ThreadVox<V>& tv,
                                            const float* slot, int (&mn)[3], int (&mx)[3]) {
    constexpr int NV = kThreads * V;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        mn[k] = INT_MAX;
        mx[k] = INT_MIN;
    }
#pragma unroll
    for (int q = 0; q < V; ++q) {
        const int lin = threadIdx.x + q * kThreads;
        if (tv.template index<IT>(o, q) < 0) continue;
        float x[3];
        if (!load_valid(slot[lin], slot[NV + lin], slot[2 * NV + lin], g, x[0], x[1], x[2])) continue;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int f = first_tap32(x[k], DP);
            const int c = f < -kClamp ? -kClamp : (f > kClamp ? kClamp : f);
            mn[k] = min(mn[k], c);
            mx[k] = max(mx[k], c);
        }
    }
}

// Planes in flight in the tiled kernels: two for pull up to four taps; the
// derivative ops, with more accumulators, and five taps one (two would need more
// registers than 16 warps per SM leave: quartic pull of 192^3 281 us spilling, 240
// with one).
template <int OP, int DP>
constexpr int kRolled = OP == kPull && DP <= 4 ? 2 : 1;

// contract_rolled over the shared box: row (k, j) starts at p + k*Q4 + j*P4.
template <int OP, int DP, class WT>
__device__ __forceinline__ void contract_smem(const WT& ax, const WT& ay, const WT& az, unsigned p, unsigned P4,
                                              unsigned Q4, float (&r)[6]) {
    contract_rolled<OP, DP, kRolled<OP, DP>>(
        ax, ay, az, [&](int j, float (&f)[DP]) { lds_row<DP>(p + j * P4, f); }, [&]() { p += Q4; }, r);
}

// pull_voxel_global (pp_voxel.cuh) for the tiles whose box does not fit, inlined
// into the tiled kernels with the rolled contraction so that it costs them no
// registers (a call, or the fully unrolled global gather, made the whole
// kernel spill).
template <int DP, int OP_, typename IT>
__device__ __forceinline__ void pull_voxel_lean(const LaunchArgs& a, int b, long long v, float x0, float x1,
                                                float x2) {
    constexpr int OP = pull_base_op<OP_>();
    constexpr int ORD = op_order(OP);
    const Geometry& g = a.g;
    const long long n1 = g.n1;
    const IT sy = (IT)g.d0[0];
    const IT sz = (IT)(g.d0[0] * g.d0[1]);
    float acc[3] = {0.f, 0.f, 0.f};
    Axis<DP, ORD, IT> ax, ay, az;
#pragma unroll 1
    for (int c = 0; c < g.nc; ++c) {
        int b0, b1, b2;
        bnd_code(a, c, b0, b1, b2);
        ax.setup(x0, g.dp[0], b0, g.d0[0], (IT)1);
        ay.setup(x1, g.dp[1], b1, g.d0[1], sy);
        az.setup(x2, g.dp[2], b2, g.d0[2], sz);
        const float* f0 = a.in + ((long long)b * g.nc + c) * g.n0;
        IT zo[DP];
#pragma unroll
        for (int i = 0; i < DP; ++i) zo[i] = az.off[i];
        float r[6];
        contract_rolled<OP, DP, kRolled<OP, DP>>(
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
        if constexpr (pull_is_dot<OP_>()) dot_accumulate<OP_>(a, b, c, v, r, acc);
        else pull_store<OP>(pull_out<OP_>(a, b, c, v), n1, r);
    }
    if constexpr (pull_is_dot<OP_>()) {
        float* o = pull_out<OP_>(a, b, 0, v);
        o[0] = acc[0];
        o[n1] = acc[1];
        o[2 * n1] = acc[2];
    }
}

// push_voxel_global (pp_voxel.cuh) for plain push, inlined with the z loop
// rolled (weights and offsets rotate through slot 0) so that the fallback of the
// batched kernel pins no registers across a call.  The values are read with
// plain loads: the batched kernel wrote them earlier in the same launch.
template <int DP, typename IT>
__device__ __forceinline__ void push_voxel_lean(const LaunchArgs& a, int b, long long v, float x0, float x1,
                                                float x2) {
    const Geometry& g = a.g;
    const long long n1 = g.n1;
    const IT sy = (IT)g.d0[0];
    const IT sz = (IT)(g.d0[0] * g.d0[1]);
#pragma unroll 1
    for (int c = 0; c < g.nc; ++c) {
        const float v0 = a.in[((long long)b * g.nc + c) * n1 + v];
        if (!finitef(v0)) continue;
        int b0, b1, b2;
        bnd_code(a, c, b0, b1, b2);
        Axis<DP, 0, IT> ax, ay, az;
        ax.setup(x0, g.dp[0], b0, g.d0[0], (IT)1);
        ay.setup(x1, g.dp[1], b1, g.d0[1], sy);
        az.setup(x2, g.dp[2], b2, g.d0[2], sz);
        float* f0 = a.out + ((long long)b * g.nc + c) * g.n0;
#pragma unroll 1
        for (int k = 0; k < DP; ++k) {
#pragma unroll
            for (int j = 0; j < DP; ++j) {
                const float cb = v0 * (ay.w[j] * az.w[0]);
#pragma unroll
                for (int i = 0; i < DP; ++i) atomicAdd(f0 + (az.off[0] + ay.off[j] + ax.off[i]), cb * ax.w[i]);
            }
#pragma unroll
            for (int i = 0; i + 1 < DP; ++i) {
                az.w[i] = az.w[i + 1];
                az.off[i] = az.off[i + 1];
            }
        }
    }
}

// A whole tile whose footprint box does not fit in shared memory: every voxel
// from global memory, all channels.
template <int DP, int OP, int V, typename IT>
__device__ __forceinline__ void pull_tile_global(const LaunchArgs& a, const TileOrigin& o, const ThreadVox<V>& tv,
                                                 const TileGrid& t, const float* slot) {
    constexpr int NV = kThreads * V;
#pragma unroll 1
    for (int q = 0; q < V; ++q) {
        const int lin = threadIdx.x + q * kThreads;
        const IT v = tv.template index_lin<IT>(o, lin, t);
        if (v < 0) continue;
        float x0, x1, x2;
        if (!load_valid(slot[lin], slot[NV + lin], slot[2 * NV + lin], a.g, x0, x1, x2))
            pull_voxel_nan<OP>(a, o.b, (long long)v);
        else
            pull_voxel_lean<DP, OP, IT>(a, o.b, (long long)v, x0, x1, x2);
    }
}

// Evaluate channel c of a tile for the pull family (dot ops accumulate into
// acc[q] and store after the last channel).
template <int DP, int OP_, int V, typename IT>
__device__ __forceinline__ void pull_compute(const LaunchArgs& a, const TileOrigin& o, const ThreadVox<V>& tv,
                                             const TileGrid& t, const float* slot, int c, const Box& box,
                                             const float* sm, float (&acc)[V][3]) {
    constexpr int OP = pull_base_op<OP_>();
    constexpr int NCOMP = pull_ncomp<OP_>();
    constexpr int NV = kThreads * V;
    const Geometry& g = a.g;
    const long long n1 = g.n1;
    const bool last = c == g.nc - 1;
    auto voxel = [&](int q) {
        const int lin = threadIdx.x + q * kThreads;
        const IT v = tv.template index_lin<IT>(o, lin, t);
        if (v < 0) return;
        float x0, x1, x2;
        if (!load_valid(slot[lin], slot[NV + lin], slot[2 * NV + lin], g, x0, x1, x2)) {
            if (!pull_is_dot<OP_>() || last) {
                float* out = pull_out<OP_>(a, o.b, c, (long long)v);
#pragma unroll
                for (int p = 0; p < NCOMP; ++p) out[(long long)p * n1] = qnan();
            }
            return;
        }
        if (box.mode != 1) return;   // mode 0: no valid voxel; mode 2 tiles never get here
        constexpr int ORD = op_order(OP);
        W3<DP, ORD> wx, wy, wz;
        const int ox = spline_taps32<DP, ORD>(x0, wx.w, wx.dw, wx.hw) - box.xo;
        const int oy = spline_taps32<DP, ORD>(x1, wy.w, wy.dw, wy.hw) - box.lo[1];
        const int oz = spline_taps32<DP, ORD>(x2, wz.w, wz.dw, wz.hw) - box.lo[2];
        const unsigned P4 = 4u * box.P, Q4 = 4u * box.Q;
        const unsigned p = smem_addr(sm) + 4u * (unsigned)(oz * box.Q + oy * box.P + ox);
        float r[6];
        contract_smem<OP, DP>(wx, wy, wz, p, P4, Q4, r);
        if constexpr (pull_is_dot<OP_>()) {
            dot_accumulate<OP_>(a, o.b, c, (long long)v, r, acc[q]);
            if (last) {
                float* out = pull_out<OP_>(a, o.b, 0, (long long)v);
                out[0] = acc[q][0];
                out[n1] = acc[q][1];
                out[2 * n1] = acc[q][2];
            }
        } else {
            pull_store<OP>(pull_out<OP_>(a, o.b, c, (long long)v), n1, r);
        }
    };
    if constexpr (pull_is_dot<OP_>()) {
        // acc[q] stays in registers only with a compile-time q
#pragma unroll
        for (int q = 0; q < V; ++q) voxel(q);
    } else {
        // one voxel at a time: interleaving the V voxels' patches needs more
        // registers than two resident CTAs per SM leave
#pragma unroll 1
        for (int q = 0; q < V; ++q) voxel(q);
    }
}

// Persistent, software-pipelined pull family.  CTA i walks tiles i, i+G, i+2G, ...
// (G = grid size).  The deformation of the next kStages tiles is in flight in the
// tile ring; while tile j is evaluated from one box buffer, the box of tile j+1
// is being staged into the other with cp.async.
template <int DP, int OP, int V, typename IT, bool TMA>
__global__ void __launch_bounds__(kThreads, 2) k_pull_tiled(const __grid_constant__ LaunchArgs a,
                                                            const __grid_constant__ TileGrid t,
                                                            const __grid_constant__ CUtensorMap phimap,
                                                            const __grid_constant__ CUtensorMap imgmap) {
    extern __shared__ __align__(128) float4 smem4[];
    constexpr int NV = kThreads * V;
    __shared__ int red[8][7];
    __shared__ Box boxm[2];
    __shared__ int s_abort;
    const Geometry& g = a.g;
    const int G = gridDim.x;
    const int T0 = blockIdx.x;
    if (T0 >= t.ntiles) return;
    const int ntl = (t.ntiles - T0 + G - 1) / G;
    const ThreadVox<V> tv(t, g);

    float* sm = reinterpret_cast<float*>(smem4);
    Ring ring;
    ring.base = sm;
    ring.slot_floats = 3 * NV;
    float* bufs = sm + kStages * 3 * NV;
    ring.bars = smem_addr(bufs + 2 * t.cap);
    const unsigned bbar = ring.bars + 8u * kStages;   // one mbarrier per box buffer (TMA-staged boxes)
    unsigned bphase = 0;                              // bit b: parity of buffer b's next TMA completion
    if (threadIdx.x == 0) {
        s_abort = 0;
        if (TMA) {
            for (int k = 0; k < kStages; ++k) mbar_init(ring.bars + 8u * k, 1);
        }
        mbar_init(bbar, 1);
        mbar_init(bbar + 8u, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    for (int j = 0; j < kStages && j < ntl; ++j)
        ring_fill<V, TMA, IT>(ring, j, T0 + j * G, a, t, tv, phimap);
    if (!TMA) __syncthreads();

    // one TMA copy of channel c's fixed image window into buffer `buf` (thread 0)
    auto tma_box = [&](const Box& box, int b, int c, int buf) {
        if (threadIdx.x == 0) {
            const unsigned bar = bbar + 8u * buf;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_expect_tx(bar, (unsigned)(kTmaBoxFloats * sizeof(float)));
            tma_load_4d(smem_addr(bufs + buf * t.cap), &imgmap, bar, box.xo, box.lo[1], box.lo[2], b * g.nc + c);
        }
    };
    // every thread: wait for buffer buf's TMA copy
    auto tma_wait = [&](int buf) {
        if (!mbar_wait(bbar + 8u * buf, (bphase >> buf) & 1u)) s_abort = 1;
        bphase ^= 1u << buf;
    };

    // box of tile j (its deformation must be in the ring), staged into buffer j & 1
    auto prepare = [&](int j) {
        const TileOrigin o = tile_origin(t, T0 + j * G);
        const float* slot = ring.base + (j % kStages) * ring.slot_floats;
        if (!ring_wait<TMA>(ring, j)) s_abort = 1;
        int mn[3], mx[3];
        tile_bounds<DP, V, IT>(g, o, tv, slot, mn, mx);
        reduce_box<DP>(mn, mx, t, g, 1, boxm[j & 1], red);
        if (boxm[j & 1].mode == 1) {
            if (boxm[j & 1].tma) {
                tma_box(boxm[j & 1], o.b, 0, j & 1);
            } else {
                int b0, b1, b2;
                bnd_code(a, 0, b0, b1, b2);
                stage_box<IT>(boxm[j & 1], g, b0, b1, b2, a.in + (long long)o.b * g.nc * g.n0,
                              bufs + (j & 1) * t.cap);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };

    prepare(0);
    for (int j = 0; j < ntl; ++j) {
        if (j + 1 < ntl) {
            prepare(j + 1);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        if (boxm[j & 1].tma) tma_wait(j & 1);   // the record was published by prepare(j)'s barrier
        __syncthreads();   // box j is in its buffer
        if (s_abort) break;
        const TileOrigin o = tile_origin(t, T0 + j * G);
        const float* slot = ring.base + (j % kStages) * ring.slot_floats;
        const Box& box = boxm[j & 1];
        float* buf = bufs + (j & 1) * t.cap;
        if (box.mode == 2) {
            pull_tile_global<DP, OP, V, IT>(a, o, tv, t, slot);
            __syncthreads();   // ring slot j is free
            if (j + kStages < ntl)
                ring_fill<V, TMA, IT>(ring, j + kStages, T0 + (j + kStages) * G, a, t, tv, phimap);
            if (!TMA) __syncthreads();
            continue;
        }
        float acc[V][3];
#pragma unroll
        for (int q = 0; q < V; ++q) acc[q][0] = acc[q][1] = acc[q][2] = 0.f;
        pull_compute<DP, OP, V, IT>(a, o, tv, t, slot, 0, box, buf, acc);
        for (int c = 1; c < g.nc; ++c) {
            __syncthreads();   // channel c-1 reads of the buffer are done
            if (box.mode == 1) {
                if (box.tma) {
                    tma_box(box, o.b, c, j & 1);
                    tma_wait(j & 1);
                } else {
                    int b0, b1, b2;
                    bnd_code(a, c, b0, b1, b2);
                    stage_box<IT>(box, g, b0, b1, b2, a.in + ((long long)o.b * g.nc + c) * g.n0, buf);
                    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
                }
            }
            __syncthreads();
            if (s_abort) break;
            pull_compute<DP, OP, V, IT>(a, o, tv, t, slot, c, box, buf, acc);
        }
        if (s_abort) break;
        __syncthreads();   // ring slot j and buffer j & 1 are free
        if (j + kStages < ntl)
            ring_fill<V, TMA, IT>(ring, j + kStages, T0 + (j + kStages) * G, a, t, tv, phimap);
        if (!TMA) __syncthreads();
    }
}

// Scatter one voxel into the push accumulator (box-relative first taps ox, oy, oz).
// FIXED: two int32 words per element (values pre-scaled to q1 units); otherwise float.
// WT: any weight set with w (and dw for push_grad) of DP taps.
template <int DP, int OP, bool FIXED, class WT>
__device__ __forceinline__ void push_scatter(const WT& wx, const WT& wy, const WT& wz, float v0, float v1, float v2,
                                             unsigned base, unsigned P4, unsigned Q4, unsigned lo_off) {
#pragma unroll
    for (int k = 0; k < DP; ++k) {
#pragma unroll
        for (int j = 0; j < DP; ++j) {
            float ca, cb;
            if constexpr (OP == kPushGrad) {
                ca = v0 * (wy.w[j] * wz.w[k]);
                cb = v1 * (wy.dw[j] * wz.w[k]) + v2 * (wy.w[j] * wz.dw[k]);
            } else {
                ca = 0.f;
                cb = v0 * (wy.w[j] * wz.w[k]);
            }
            const unsigned row = base + k * Q4 + j * P4;
            if constexpr (FIXED) {
                int h[DP], l[DP];
                // taps in pairs with the packed f32x2 pipe (each lane rounds exactly
                // like the scalar sequence of the odd tap below)
#pragma unroll
                for (int i = 0; i + 1 < DP; i += 2) {
                    float2 y2;
                    if constexpr (OP == kPushGrad)
                        y2 = __ffma2_rn(make_float2(ca, ca), make_float2(wx.dw[i], wx.dw[i + 1]),
                                        __fmul2_rn(make_float2(cb, cb), make_float2(wx.w[i], wx.w[i + 1])));
                    else
                        y2 = __fmul2_rn(make_float2(cb, cb), make_float2(wx.w[i], wx.w[i + 1]));
                    const float2 t1 = __fadd2_rn(y2, make_float2(kMagic, kMagic));
                    const float2 u = __fadd2_rn(t1, make_float2(-kMagic, -kMagic));
                    const float2 r = __ffma2_rn(u, make_float2(-1.f, -1.f), y2);
                    const float2 l2 = __ffma2_rn(r, make_float2(kLoScale, kLoScale), make_float2(kMagic, kMagic));
                    h[i] = __float_as_int(t1.x) - kMagicBits;
                    h[i + 1] = __float_as_int(t1.y) - kMagicBits;
                    l[i] = __float_as_int(l2.x) - kMagicBits;
                    l[i + 1] = __float_as_int(l2.y) - kMagicBits;
                }
                if constexpr (DP & 1) {
                    constexpr int i = DP - 1;
                    float y;
                    if constexpr (OP == kPushGrad) y = fmaf(ca, wx.dw[i], cb * wx.w[i]);
                    else y = cb * wx.w[i];
                    // y in q1 units, |y| <= 2^22: hi = round(y), lo = round((y - hi) * 2^21)
                    const float t1 = __fadd_rn(y, kMagic);
                    const float r = __fsub_rn(y, __fsub_rn(t1, kMagic));
                    h[i] = __float_as_int(t1) - kMagicBits;
                    l[i] = __float_as_int(__fmaf_rn(r, kLoScale, kMagic)) - kMagicBits;
                }
                red_row_s32<DP>(row, h);
                red_row_s32<DP>(row + lo_off, l);
            } else {
#pragma unroll
                for (int i = 0; i < DP; ++i) {
                    float y;
                    if constexpr (OP == kPushGrad) y = fmaf(ca, wx.dw[i], cb * wx.w[i]);
                    else y = cb * wx.w[i];
                    red_shared_f32(row + 4u * i, y);
                }
            }
        }
    }
}

// Shared-memory reductions without a compiler memory barrier, so that loads of
// the next voxels can be issued ahead of them (what they read and the
// accumulator are disjoint; the phases are separated by __syncthreads).
__device__ __forceinline__ void red_s32_nb(unsigned a, int v) {
    asm volatile("red.shared.add.s32 [%0], %1;" ::"r"(a), "r"(v));
}
__device__ __forceinline__ void red_f32_nb(unsigned a, float v) {
    asm volatile("red.shared.add.f32 [%0], %1;" ::"r"(a), "f"(v));
}

#ifdef PP_TILED_BATCH
// ---- batched uneven workload ------------------------------------------------
//
// Tiles of all items form one queue; a CTA takes the next tile with an atomic
// counter (dynamic load balance over volumes of uneven size and degree),
// evaluates pull for the tile from its staged image box, writes f1, and pushes
// the same values through the same box into the shared accumulator, which it
// flushes into the item's output.  Shared memory is split into a fixed
// accumulator region (two words per element) and the image box.

template <int DP>
__device__ __forceinline__ void batch_tile(const BatchItem& it, int lt, float* sm, int cap, Box& box,
                                           int (&red)[8][7], float (&sred)[8]) {
    constexpr int V = 2;
    constexpr int NV = kThreads * V;
    const LaunchArgs& a = it.pull;
    const LaunchArgs& pb = it.push;
    const Geometry& g = a.g;
    const long long n1 = g.n1;
    const TileGrid& t = it.t;
    const ThreadVox<V> tv(t, g);
    const TileOrigin o = tile_origin(t, lt);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int accw = ((2 * cap / 3) + 3) & ~3;   // accumulator words (fixed region)
    float* accf = sm;
    float* fbox = sm + accw;

    float X[V][3];
    int iv[V];
    unsigned ok = 0;
    int mn[3] = {INT_MAX, INT_MAX, INT_MAX}, mx[3] = {INT_MIN, INT_MIN, INT_MIN};
#pragma unroll
    for (int q = 0; q < V; ++q) {
        iv[q] = tv.template index<int>(o, q);
        if (iv[q] < 0) continue;
        const float* phi = a.phi + iv[q];
        if (!load_valid(__ldg(phi), __ldg(phi + n1), __ldg(phi + 2 * n1), g, X[q][0], X[q][1], X[q][2])) continue;
        ok |= 1u << q;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int f = first_tap32(X[q][k], DP);
            const int cl = f < -kClamp ? -kClamp : (f > kClamp ? kClamp : f);
            mn[k] = min(mn[k], cl);
            mx[k] = max(mx[k], cl);
        }
    }
    reduce_box<DP>(mn, mx, t, g, 3, box, red);   // 3 words per element: 2 accumulator + 1 image
    if (box.mode != 1) {
#pragma unroll
        for (int q = 0; q < V; ++q) {
            if (iv[q] < 0) continue;
            if (!(ok >> q & 1)) {
                pull_voxel_nan<kPull>(a, 0, iv[q]);
                continue;
            }
            pull_voxel_lean<DP, kPull, int>(a, 0, iv[q], X[q][0], X[q][1], X[q][2]);
            push_voxel_lean<DP, int>(pb, 0, iv[q], X[q][0], X[q][1], X[q][2]);
        }
        __syncthreads();   // box record reused by the next tile
        return;
    }
    const unsigned acc_base = smem_addr(accf);
    const unsigned lo_off = 4u * (unsigned)box.size;
    int* acc_hi = reinterpret_cast<int*>(accf);
    int* acc_lo = acc_hi + box.size;
    for (int c = 0; c < g.nc; ++c) {
        int b0, b1, b2;
        bnd_code(a, c, b0, b1, b2);
        stage_box<int>(box, g, b0, b1, b2, a.in + (long long)c * g.n0, fbox);
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
        float val[V];
        float bound = 0.f;
        float* f1 = a.out + (long long)c * n1;
#pragma unroll
        for (int q = 0; q < V; ++q) {
            val[q] = 0.f;
            if (iv[q] < 0) continue;
            if (!(ok >> q & 1)) {
                f1[iv[q]] = qnan();
                continue;
            }
            W3<DP, 0> wx, wy, wz;
            const int ox = spline_taps32<DP, 0>(X[q][0], wx.w, wx.dw, wx.hw) - box.xo;
            const int oy = spline_taps32<DP, 0>(X[q][1], wy.w, wy.dw, wy.hw) - box.lo[1];
            const int oz = spline_taps32<DP, 0>(X[q][2], wz.w, wz.dw, wz.hw) - box.lo[2];
            const unsigned P4 = 4u * box.P, Q4 = 4u * box.Q;
            const unsigned p = smem_addr(fbox) + 4u * (unsigned)(oz * box.Q + oy * box.P + ox);
            float r[6];
            contract_smem<kPull, DP>(wx, wy, wz, p, P4, Q4, r);
            f1[iv[q]] = r[0];
            val[q] = r[0];
            if (finitef(r[0])) bound += fabsf(r[0]);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) bound += __shfl_xor_sync(0xffffffffu, bound, off);
        if (lane == 0) sred[warp] = bound;
        __syncthreads();   // bounds in; the image box is no longer read
        float S = 0.f;
        for (int w = 0; w < kThreads / 32; ++w) S += sred[w];
        const int E = scale_exponent(S);
        if (E != INT_MAX) {
            const bool fixed = E != INT_MIN;
            FixedScale fs;
            fs.set(fixed ? E : 0);
#pragma unroll
            for (int q = 0; q < V; ++q) {
                if (!(ok >> q & 1) || !finitef(val[q])) continue;
                W3<DP, 0> wx, wy, wz;
                const int ox = spline_taps32<DP, 0>(X[q][0], wx.w, wx.dw, wx.hw) - box.xo;
                const int oy = spline_taps32<DP, 0>(X[q][1], wy.w, wy.dw, wy.hw) - box.lo[1];
                const int oz = spline_taps32<DP, 0>(X[q][2], wz.w, wz.dw, wz.hw) - box.lo[2];
                const unsigned P4 = 4u * box.P, Q4 = 4u * box.Q;
                const unsigned base = acc_base + 4u * (unsigned)(oz * box.Q + oy * box.P + ox);
                if (fixed) push_scatter<DP, kPush, true>(wx, wy, wz, val[q] * fs.inv_q1, 0.f, 0.f, base, P4, Q4, lo_off);
                else push_scatter<DP, kPush, false>(wx, wy, wz, val[q], 0.f, 0.f, base, P4, Q4, lo_off);
            }
            __syncthreads();   // the scatter is complete
            float* out = pb.out + (long long)c * g.n0;
            if (fixed)
                flush_box<int>(box, g, b0, b1, b2, out, [&](int si) {
                    const float v = fixed_value(acc_hi[si], acc_lo[si], fs);
                    acc_hi[si] = 0;
                    acc_lo[si] = 0;
                    return v;
                });
            else
                flush_box<int>(box, g, b0, b1, b2, out, [&](int si) {
                    const float v = accf[si];
                    accf[si] = 0.f;
                    return v;
                });
        }
        __syncthreads();   // accumulator clear, image box and sred reusable
    }
}

// A tile of an item with per-dimension degrees: every voxel from global memory
// (runtime degree per axis), each channel pulled and its value pushed straight
// back with global atomics.
__device__ __noinline__ void batch_tile_any(const BatchItem& it, int lt) {
    constexpr int V = 2;
    const LaunchArgs& a = it.pull;
    const Geometry& g = a.g;
    const long long n1 = g.n1;
    const TileGrid& t = it.t;
    const ThreadVox<V> tv(t, g);
    const TileOrigin o = tile_origin(t, lt);
    const int sy = (int)g.d0[0], sz = (int)(g.d0[0] * g.d0[1]);
#pragma unroll 1
    for (int q = 0; q < V; ++q) {
        const int v = tv.template index<int>(o, q);
        if (v < 0) continue;
        const float* phi = a.phi + v;
        float x0, x1, x2;
        if (!load_valid(__ldg(phi), __ldg(phi + n1), __ldg(phi + 2 * n1), g, x0, x1, x2)) {
            pull_voxel_nan<kPull>(a, 0, v);
            continue;
        }
        Axis<0, 0, int> ax, ay, az;
        constexpr int N = Axis<0, 0, int>::N;
        int prev = -1;
#pragma unroll 1
        for (int c = 0; c < g.nc; ++c) {
            int b0, b1, b2;
            const int code = bnd_code(a, c, b0, b1, b2);
            if (code != prev) {
                ax.setup(x0, g.dp[0], b0, g.d0[0], 1);
                ay.setup(x1, g.dp[1], b1, g.d0[1], sy);
                az.setup(x2, g.dp[2], b2, g.d0[2], sz);
                prev = code;
            }
            const float* f0 = a.in + (long long)c * g.n0;
            float r[6];
            contract<kPull, N>(ax, ay, az, ax.n, ay.n, az.n,
                               [&](int k, int j, int i) { return __ldg(f0 + (az.off[k] + ay.off[j] + ax.off[i])); }, r);
            a.out[(long long)c * n1 + v] = r[0];
            if (!finitef(r[0])) continue;
            float* out = it.push.out + (long long)c * g.n0;
#pragma unroll 1
            for (int k = 0; k < az.n; ++k) {
#pragma unroll 1
                for (int j = 0; j < ay.n; ++j) {
                    const float cb = r[0] * (ay.w[j] * az.w[k]);
                    float* row = out + (az.off[k] + ay.off[j]);
#pragma unroll 1
                    for (int i = 0; i < ax.n; ++i) atomicAdd(row + ax.off[i], cb * ax.w[i]);
                }
            }
        }
    }
}

__global__ void __launch_bounds__(kThreads, 2) k_batch(const BatchItem* __restrict__ items, int nitems, int total,
                                                       unsigned* counter, int cap) {
    extern __shared__ __align__(128) float4 smem4[];
    __shared__ int red[8][7];
    __shared__ float sred[8];
    __shared__ Box box;
    __shared__ int s_tile;
    float* sm = reinterpret_cast<float*>(smem4);
    const int accw = ((2 * cap / 3) + 3) & ~3;
    for (int i = threadIdx.x; i < (accw >> 2); i += kThreads)
        reinterpret_cast<float4*>(sm)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (;;) {
        if (threadIdx.x == 0) s_tile = (int)atomicAdd(counter, 1u);
        __syncthreads();
        const int T = s_tile;
        __syncthreads();   // every thread has read the tile before the next claim
        if (T >= total) break;
        int lo = 0, hi = nitems - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (items[mid].tile_begin <= T) lo = mid;
            else hi = mid - 1;
        }
        const BatchItem& it = items[lo];
        const int lt = T - it.tile_begin;
        switch (it.dp) {
            case 0: batch_tile_any(it, lt); break;
            case 1: batch_tile<1>(it, lt, sm, cap, box, red, sred); break;
            case 2: batch_tile<2>(it, lt, sm, cap, box, red, sred); break;
            case 3: batch_tile<3>(it, lt, sm, cap, box, red, sred); break;
            case 4: batch_tile<4>(it, lt, sm, cap, box, red, sred); break;
            default: batch_tile<5>(it, lt, sm, cap, box, red, sred); break;
        }
    }
}
#endif  // PP_TILED_BATCH

TileGrid make_grid(const LaunchArgs& a, const TileCfg& c) {
    TileGrid t;
    t.lx = c.lx;
    t.ly = c.ly;
    t.lz = c.lz;
    t.ntx = (int)((a.g.d1[0] + (1 << c.lx) - 1) >> c.lx);
    t.nty = (int)((a.g.d1[1] + (1 << c.ly) - 1) >> c.ly);
    t.ntz = (int)((a.g.d1[2] + (1 << c.lz) - 1) >> c.lz);
    t.cap = c.cap;
    t.ntiles = t.ntx * t.nty * t.ntz * a.g.nb;
    auto magic = [](int d, unsigned long long& m, int& sh) {
        int l = 0;
        while ((1LL << l) < d) ++l;                        // l = ceil(log2 d)
        sh = 31 + l;
        m = ((1ULL << sh) + (unsigned long long)d - 1) / (unsigned long long)d;
    };
    magic(t.ntx, t.mx, t.sx);
    magic(t.nty, t.my, t.sy);
    magic(t.ntz, t.mz, t.sz);
    const int tx = 1 << c.lx;
    t.pmod = tx >= 32 ? 0 : tx;
    t.img_tma = t.phi_tma = t.winy = t.winz = 0;
    t.nv = tx << (c.ly + c.lz);
    t.stages = 0;
    return t;
}

// Raise a kernel's dynamic shared-memory limit once per (device, kernel) to the
// largest size requested so far.
template <typename K>
cudaError_t opt_in(K kern, size_t smem) {
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, size_t> configured;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const auto key = std::make_pair(dev, reinterpret_cast<const void*>(kern));
    std::lock_guard<std::mutex> lk(mu);
    auto it = configured.find(key);
    if (it != configured.end() && it->second >= smem) return cudaSuccess;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    configured[key] = smem;
    return cudaSuccess;
}

// ---- TMA tensor maps (encoded on the host through the driver entry point) ----
using EncodeFn = PFN_cuTensorMapEncodeTiled_v12000;

EncodeFn encode_fn() {
    static std::once_flag once;
    static EncodeFn fn = nullptr;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeFn>(p);
    });
    return fn;
}

// 4-D map over a column-major volume stack (d0, d1, d2, planes) with a box of
// one tile (TX, TY, TZ, comps).  Requires a 16-byte aligned base and d0 % 4 == 0.
bool encode_tile_map(CUtensorMap* map, const float* base, const long long d[3], long long planes,
                     const TileGrid& t, int comps) {
    EncodeFn fn = encode_fn();
    if (!fn) return false;
    if ((reinterpret_cast<uintptr_t>(base) & 15) || (d[0] & 3) || (1 << t.lx) < 4) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)d[0], (cuuint64_t)d[1], (cuuint64_t)d[2], (cuuint64_t)planes};
    for (int k = 0; k < 4; ++k)
        if (dims[k] == 0 || dims[k] > (1ULL << 32)) return false;
    const cuuint64_t strides[3] = {(cuuint64_t)d[0] * 4, (cuuint64_t)(d[0] * d[1]) * 4,
                                   (cuuint64_t)(d[0] * d[1] * d[2]) * 4};
    for (int k = 0; k < 3; ++k)
        if (strides[k] >= (1ULL << 40)) return false;
    const cuuint32_t box[4] = {(cuuint32_t)(1 << t.lx), (cuuint32_t)(1 << t.ly), (cuuint32_t)(1 << t.lz),
                               (cuuint32_t)comps};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

// Tensor map of an image (d0[0], d0[1], d0[2], planes) with the fixed
// kTmaBox* window as its box; false when TMA cannot address it (base or row
// stride not 16-byte aligned, dimensions out of range).
bool encode_box_map(CUtensorMap* map, const float* base, const long long d[3], long long planes) {
    auto fn = encode_fn();
    if (!fn) return false;
    if ((reinterpret_cast<uintptr_t>(base) & 15) || (d[0] & 3)) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)d[0], (cuuint64_t)d[1], (cuuint64_t)d[2], (cuuint64_t)planes};
    for (int k = 0; k < 4; ++k)
        if (dims[k] == 0 || dims[k] > (1ULL << 32)) return false;
    const cuuint64_t strides[3] = {(cuuint64_t)d[0] * 4, (cuuint64_t)(d[0] * d[1]) * 4,
                                   (cuuint64_t)(d[0] * d[1] * d[2]) * 4};
    for (int k = 0; k < 3; ++k)
        if (strides[k] >= (1ULL << 40)) return false;
    const cuuint32_t box[4] = {(cuuint32_t)kTmaBoxX, (cuuint32_t)kTmaBoxY, (cuuint32_t)kTmaBoxZ, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

// Resident CTAs per SM of a kernel with `smem` bytes of dynamic shared memory,
// asked of the runtime once per (device, kernel, size).
template <typename K>
cudaError_t resident_ctas(K kern, int threads, size_t smem, int* per_sm) {
    static std::mutex mu;
    static std::map<std::pair<std::pair<int, const void*>, size_t>, int> known;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const auto key = std::make_pair(std::make_pair(dev, reinterpret_cast<const void*>(kern)), smem);
    std::lock_guard<std::mutex> lk(mu);
    auto it = known.find(key);
    if (it == known.end()) {
        int n = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, smem);
        if (e != cudaSuccess) return e;
        it = known.emplace(key, n < 1 ? 1 : n).first;
    }
    *per_sm = it->second;
    return cudaSuccess;
}

template <typename K, typename... Args>
cudaError_t launch_persistent(K kern, const TileGrid& t, size_t smem, cudaStream_t s, int threads,
                              const Args&... args) {
    cudaError_t e = opt_in(kern, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = resident_ctas(kern, threads, smem, &per_sm);
    if (e != cudaSuccess) return e;
    const long long want = (long long)sm_count() * per_sm;
    const int grid = (int)(t.ntiles < want ? t.ntiles : want);
    kern<<<grid, threads, smem, s>>>(args...);
    return cudaGetLastError();
}

template <int DP, int OP, int V, typename IT>
cudaError_t launch_v(const LaunchArgs& a, const TileGrid& t, cudaStream_t s) {
    constexpr int NV = kThreads * V;
    CUtensorMap phimap, imgmap;
    std::memset(&phimap, 0, sizeof phimap);
    std::memset(&imgmap, 0, sizeof imgmap);
    const long long nb = a.g.nb, nc = a.g.nc;
    const bool tma = encode_tile_map(&phimap, a.phi, a.g.d1, 3 * nb, t, 3);
    // interior boxes as one TMA copy of a fixed window when the tile is 8 wide
    // (the window's row pitch is bank-conflict free for 8-wide warp tiles)
    TileGrid tt = t;
    tt.img_tma = t.lx == 3 && t.cap >= kTmaBoxFloats && (t.cap & 31) == 0 &&
                 encode_box_map(&imgmap, a.in, a.g.d0, nc * nb);
    const size_t smem = (size_t)kStages * 3 * NV * 4 + 2 * (size_t)t.cap * 4 + 8 * kStages + 16;
    if (tma) return launch_persistent(k_pull_tiled<DP, OP, V, IT, true>, tt, smem, s, kThreads, a, tt, phimap, imgmap);
    return launch_persistent(k_pull_tiled<DP, OP, V, IT, false>, tt, smem, s, kThreads, a, tt, phimap, imgmap);
}

template <int DP, int OP, typename IT>
cudaError_t launch_one(const LaunchArgs& a, const TileCfg& c, cudaStream_t s) {
    const TileGrid t = make_grid(a, c);
    if (t.nv > kThreads) return launch_v<DP, OP, 2, IT>(a, t, s);
    return launch_v<DP, OP, 1, IT>(a, t, s);
}

template <int OP, typename IT>
cudaError_t dispatch(const LaunchArgs& a, const TileCfg& t, cudaStream_t s) {
    switch (a.g.dp[0]) {
        case 1: return launch_one<1, OP, IT>(a, t, s);
        case 2: return launch_one<2, OP, IT>(a, t, s);
        case 3: return launch_one<3, OP, IT>(a, t, s);
        case 4: return launch_one<4, OP, IT>(a, t, s);
        default: return launch_one<5, OP, IT>(a, t, s);
    }
}

}  // namespace
}  // namespace pp
