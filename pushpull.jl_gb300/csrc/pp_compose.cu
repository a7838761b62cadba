// pp_compose.cu -- one step of the exponential of a velocity field: a displacement
// resampled at the positions it displaces to, u' = u o (id + u), in one pass.
//
// The reference builds id + u, then pulls u at it (src/compositions.jl:26-50):
// degree 1, extrapolated, component k with a DST-II boundary along axis k and
// DCT-II along the other two.  Here the kernel adds the identity to the
// displacement it has just read (rounded as the sum would be), so the positions
// are never stored, and the last step of the chain adds the identity to the
// result.  One thread per voxel reads its displacement coalesced and gathers the
// eight taps of the three components; mirrored taps and their signs come from a
// few selects, so voxels at the border do not leave their warp.
// What bounds it is the L1 wavefronts of the 24 gathers.  Exp of 128^3, eight
// steps, GB300: 240 us per call; 584 us as id + u and a three-channel pull per step.
#include "pp_voxel.cuh"
#include "pushpull_gb300.h"

namespace pp {
int fail_status(int code, const char* fmt, ...);

namespace {

// Signed weights and folded offsets of one axis (two taps, mirror folding).
struct MirrorAxis {
    float w[2], sw[2];   // weights; weights with the DST-II signs
    int off[2];
};

// Taps more than one period away (any finite position).
__device__ __noinline__ int mirror_far(float fo, int i, int d, float* sign) {
    return (int)fold_tap(2, (long long)fo + i, d, *sign);
}

__device__ __forceinline__ void mirror_axis(float x, int d, int stride, MirrorAxis& a) {
    const float fo = spline_weights<2, 0>(x, a.w, nullptr, nullptr);
    const bool near = fo >= -(float)d && fo + 1.0f < 2.0f * (float)d;
    const int o = near ? (int)fo : 0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        int t = o + i;
        float s = 1.0f;
        if (near) {
            const bool out = t < 0 || t >= d;
            s = out ? -1.0f : 1.0f;
            t = t < 0 ? -1 - t : (out ? 2 * d - 1 - t : t);
        } else {
            t = mirror_far(fo, i, d, &s);
        }
        a.off[i] = t * stride;
        a.sw[i] = a.w[i] * s;
    }
}

struct AxisW {
    float w[2], dw[1], hw[1];
};

template <bool ADD_ID>
__global__ void __launch_bounds__(256) k_compose_step(float* __restrict__ out, const float* __restrict__ u, int d0,
                                                      int d1, int d2) {
    const int plane = d0 * d1;
    const int p = blockIdx.x * 256 + threadIdx.x;
    if (p >= plane) return;
    const int gy = p / d0, gx = p - gy * d0;
    const long long n = (long long)plane * d2;
    const float ix = (float)(gx + 1), iy = (float)(gy + 1);
    for (int gz = blockIdx.y; gz < d2; gz += gridDim.y) {
        const long long v = (long long)gz * plane + p;
        const float iz = (float)(gz + 1);
        const float x = __fsub_rn(__fadd_rn(ix, __ldg(u + v)), 1.0f);
        const float y = __fsub_rn(__fadd_rn(iy, __ldg(u + v + n)), 1.0f);
        const float z = __fsub_rn(__fadd_rn(iz, __ldg(u + v + 2 * n)), 1.0f);
        float r[3];
        if (finitef(x) && finitef(y) && finitef(z)) {
            MirrorAxis ax, ay, az;
            mirror_axis(x, d0, 1, ax);
            mirror_axis(y, d1, d0, ay);
            mirror_axis(z, d2, plane, az);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float* f = u + c * n;
                AxisW wx, wy, wz;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    wx.w[i] = c == 0 ? ax.sw[i] : ax.w[i];
                    wy.w[i] = c == 1 ? ay.sw[i] : ay.w[i];
                    wz.w[i] = c == 2 ? az.sw[i] : az.w[i];
                }
                int k = 0;
                float q[6];
                contract_rolled<kPull, 2, 2>(
                    wx, wy, wz,
                    [&](int j, float(&t)[2]) {
                        t[0] = __ldg(f + (az.off[k] + ay.off[j] + ax.off[0]));
                        t[1] = __ldg(f + (az.off[k] + ay.off[j] + ax.off[1]));
                    },
                    [&]() { ++k; }, q);
                r[c] = q[0];
            }
        } else {
            r[0] = r[1] = r[2] = qnan();
        }
        out[v] = ADD_ID ? __fadd_rn(r[0], ix) : r[0];
        out[v + n] = ADD_ID ? __fadd_rn(r[1], iy) : r[1];
        out[v + 2 * n] = ADD_ID ? __fadd_rn(r[2], iz) : r[2];
    }
}

}  // namespace
}  // namespace pp

extern "C" int pp_compose_step(float* out, const float* u, const pp_usize d[3], int add_id, void* stream) {
    if (!d) return pp::fail_status(PP_ERR_NULL, "d must not be NULL");
    long long n = 1;
    for (int k = 0; k < 3; ++k) {
        if (d[k] >= (1ULL << 24)) return pp::fail_status(PP_ERR_TOO_LARGE, "dimension %d is 2^24 or more", k);
        n *= (long long)d[k];
        if (n >= (1LL << 31) - 1) return pp::fail_status(PP_ERR_TOO_LARGE, "volume of 2^31 voxels or more");
    }
    if (n == 0) return PP_OK;
    if (!out || !u) return pp::fail_status(PP_ERR_NULL, "data pointers must not be NULL");
    if (((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(u)) & 3) != 0)
        return pp::fail_status(PP_ERR_ALIGN, "float pointers must be 4-byte aligned");
    const dim3 grid((unsigned)((d[0] * d[1] + 255) / 256), (unsigned)(d[2] < 65535 ? d[2] : 65535));
    cudaStream_t s = (cudaStream_t)stream;
    if (add_id) pp::k_compose_step<true><<<grid, 256, 0, s>>>(out, u, (int)d[0], (int)d[1], (int)d[2]);
    else pp::k_compose_step<false><<<grid, 256, 0, s>>>(out, u, (int)d[0], (int)d[1], (int)d[2]);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PP_OK : pp::fail_status(PP_ERR_CUDA, "compose step launch: %s", cudaGetErrorString(e));
}
