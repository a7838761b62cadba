// pp_kernels.cuh -- launch descriptors and host-side launchers shared by the .cu files.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "pp_common.cuh"

namespace pp {

// kPullGradDot / kPullHessDot contract the gradient / Hessian of every channel
// with a per-voxel upstream array and sum over channels (the deformation
// cotangents of the reference rrules, src/pushpull_pb.jl:11-51).
// kPullValGrad (internal) evaluates value and gradient in one contraction.
enum PullOp { kPull = 0, kPullGrad = 1, kPullHess = 2, kPullGradDot = 3, kPullHessDot = 4, kPullValGrad = 5 };

// derivative order of the weights an op needs
__host__ __device__ constexpr int op_order(int op) {
    return op == kPull ? 0 : (op == kPullHess || op == kPullHessDot ? 2 : 1);
}
enum PushOp { kPush = 0, kPushGrad = 1 };
enum Sample { kIfBoxesFit = 1, kIfBoxesOverflow = 2 };

// Sample tile of the warp-specialised pull kernels (8 x 16 x 15 voxels) and the floats
// of its footprint box's buffer.
constexpr int kWsLy = 4, kWsTy = 1 << kWsLy, kWsTz = 15;
constexpr int kWsWinX = 24, kWsRows = 640;
constexpr int kWsCap = kWsWinX * kWsRows;

// Arguments of one pull-family or push-family launch.  Pointers address the
// first (channel 0, batch 0) element; channel c / batch b slices follow the
// reference layout (src/pushpull_cpu.jl:48, 103, 143, 198, 254).
struct LaunchArgs {
    const float* phi;   // (d1, 3, nb)
    const float* in;    // pull: f0 (d0, nc, nb); push: f1 (d1, nc, nb); push_grad: g1 (d1, 3, nc, nb)
    float* out;         // pull: (d1, ncomp, nc, nb); push: (d0, nc, nb); dot ops: (d1, 3, nb)
    const float* up;    // dot ops: upstream, (d1, nc, nb) for GradDot, (d1, 3, nc, nb) for HessDot;
                        // fused step: the target g, (d1, nc, nb)
    float* out2;        // fused step: deformation cotangent (d1, 3, nb); push: count image or NULL
    double* partial;    // fused step: one loss partial per CTA
    int sample;         // pull family: 0 always run; kIfBoxesFit, kIfBoxesOverflow: only where a sample of
                        // the deformation says so (sampled_overflow)
    Geometry g;
    BndTable bnd;
};

// Image voxels per sample voxel along the axis where they are fewest.  A sample grid
// that spans the image has about this spacing; a slab or a block of a larger grid,
// which spans a part of the image along some axes only, has it too.
inline double grid_zoom(const LaunchArgs& a) {
    double z = 1e30;
    for (int k = 0; k < 3; ++k)
        if (a.g.d1[k] > 1) {
            const double r = (double)(a.g.d0[k] - 1) / (double)(a.g.d1[k] - 1);
            z = r < z ? r : z;
        }
    return z < 1e30 ? z : 1.0;
}

// pull family: direct gather (one thread per sample voxel, all channels per thread)
cudaError_t launch_pull_direct(int op, const LaunchArgs& a, cudaStream_t s);
// push family: direct scatter with global float atomics
cudaError_t launch_push_direct(int op, const LaunchArgs& a, cudaStream_t s);

// fused forward + adjoint step, per-voxel variant (one loss partial per CTA into
// a.partial, fused_direct_grid(a).x * .y slots) and the final partial sum
dim3 fused_direct_grid(const LaunchArgs& a);
cudaError_t launch_fused_direct(const LaunchArgs& a, cudaStream_t s);
cudaError_t launch_sum_partials(const double* partial, int n, double* out, cudaStream_t s);
// Stream-ordered scratch from a pool owned by this library (one per device), freed
// with cudaFreeAsync.  The pool keeps up to kScratchKeep bytes between calls, gives the
// rest back when the stream is next synchronised, and all that is free when the
// caller asks (pp_release_scratch).  Nothing larger than kScratchMost is asked for.
// (A cubic pull of an odd volume copied through the pool, waited for after each call, us:
// 181x217x181, 27 MiB, kept 192, remapped in every call 353, without the copy 273;
// 257^3 x 2, 130 MiB, kept 697, remapped 976, without the copy 1114.)
constexpr size_t kScratchKeep = 64u << 20, kScratchMost = 256u << 20;
cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s);

// number of SMs of the current device (cached per device)
int sm_count();

}  // namespace pp
