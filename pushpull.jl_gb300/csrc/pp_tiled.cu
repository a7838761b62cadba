// pp_tiled.cu -- host side of the tiled kernels: support test, grid shape, dispatch to the
// per-group translation units and the combined device status
// (kernels and helpers: pp_tiled_impl.cuh).
#include "pp_tiled_impl.cuh"

namespace pp {

cudaError_t launch_tiled_pull_basic(int op, const LaunchArgs& a, const TileCfg& t, cudaStream_t s);
cudaError_t launch_tiled_pull_hess(int op, const LaunchArgs& a, const TileCfg& t, cudaStream_t s);
cudaError_t launch_tiled_pull_dot(int op, const LaunchArgs& a, const TileCfg& t, cudaStream_t s);
cudaError_t launch_tiled_push(int op, const LaunchArgs& a, const TileCfg& t, cudaStream_t s);
cudaError_t launch_tiled_push_grad(int op, const LaunchArgs& a, const TileCfg& t, cudaStream_t s);
unsigned status_pull_basic(bool reset);
unsigned status_pull_hess(bool reset);
unsigned status_pull_dot(bool reset);
unsigned status_push(bool reset);
unsigned status_push_grad(bool reset);
unsigned status_fused(bool reset);
unsigned status_batch(bool reset);
unsigned status_ws_pull(bool reset);
unsigned status_ws_hess(bool reset);
unsigned status_ws_grad_dot(bool reset);
unsigned status_ws_hess_dot(bool reset);
unsigned status_push_affine(bool reset);

namespace {
bool grid_supported(const LaunchArgs& a, const TileCfg& t, int max_vox) {
    const Geometry& g = a.g;
    const int vox = 1 << (t.lx + t.ly + t.lz);
    if (!(g.dp[0] == g.dp[1] && g.dp[1] == g.dp[2])) return false;
    // whole tiles of a multiple of the CTA's threads
    if (vox < kThreads || vox > max_vox || t.cap < 64 || (t.cap & 3) || t.cap > 24 * 1024) return false;
    // a tile must be mostly inside the sample grid: degenerate grids (e.g. a
    // flat list of n1 samples) are better served by the per-voxel kernels
    for (int k = 0; k < 3; ++k) {
        const int l = k == 0 ? t.lx : (k == 1 ? t.ly : t.lz);
        if (2 * g.d1[k] < (1LL << l)) return false;
    }
    const long long ntx = (g.d1[0] + (1 << t.lx) - 1) >> t.lx;
    const long long nty = (g.d1[1] + (1 << t.ly) - 1) >> t.ly;
    const long long ntz = (g.d1[2] + (1 << t.lz) - 1) >> t.lz;
    return ntx * nty * ntz * g.nb < 0x7fffffffLL;
}
}  // namespace

bool tiled_supported(const LaunchArgs& a, const TileCfg& t) { return grid_supported(a, t, 2 * kThreads); }
bool push_supported(const LaunchArgs& a, const TileCfg& t) { return grid_supported(a, t, 4 * kThreads); }

// The own tile is 16 voxels wide.  On narrow grids the per-voxel kernels are faster
// (us, per-voxel / tiled: 6x300x300 quadratic 45 / 106, cubic 82 / 152, quartic 154 / 190;
// 12x300x300 73 / 105, 149 / 152, 279 / 225).
bool fused_supported(const LaunchArgs& a, const TileCfg& t) {
    const long long x = a.g.d1[0];
    return tiled_supported(a, t) && !(t.automatic && (x <= 8 || (x < 16 && a.g.dp[0] == 3)));
}

// Push tiles: 8x8x8 voxels where they give every SM a few, else 8x8x4, so that more CTAs
// take part; budgets (accumulator words, two per element) that leave room for four CTAs
// per SM with one ring slot (push_grad at degrees 2 and 3: the ring holds three values).
// GB300, us, 8x8x8 / 8x8x4: cubic 32^3 20 / 18, 48^3 22 / 19, 64^3 29 / 28, 72^3 33 / 31,
// 80^3 37 / 37; quartic 64^3 43 / 35; quadratic 64^3 18 / 20; push_grad cubic 56^3 25 / 23,
// 72^3 33 / 32.  192^3 cubic, with the best budget of each: 8x8x8 335, 16x8x4 349, 8x16x4
// 352, 16x8x8 378.  Budgets: quadratic 192^3 9472 words 202, 11008 209; quartic 160^3
// 9472 397, 11008 344; cubic contracted 256^3 x 3 9472 1997, 11008 1751; push_grad
// 181x217x181 cubic 8448 394, 9472 427, quartic 128^3 8448 182, 9472 167.
// Grids under 8 voxels in x fill half a tile: at degree 2 the per-voxel kernels
// (6x300x300 32 / 49 us).
TileCfg push_default_tile(int op, const LaunchArgs& a) {
    const int dp = a.g.dp[0];
    if (dp == 3 && a.g.d1[0] < 8) return TileCfg{3, 3, 3, 0};
    const int cap = op == kPush ? (dp <= 3 ? 9472 : 11008) : (dp <= 4 ? 8448 : 9472);
    const long long tiles = ((a.g.d1[0] + 7) >> 3) * ((a.g.d1[1] + 7) >> 3) * ((a.g.d1[2] + 7) >> 3) * a.g.nb;
    return TileCfg{3, 3, tiles >= (dp <= 3 ? 3LL : 5LL) * sm_count() ? 3 : 2, cap};
}

cudaError_t launch_pull_tiled(int op, const LaunchArgs& a, const TileCfg& t, cudaStream_t s) {
    switch (op) {
        case kPull:
        case kPullGrad: return launch_tiled_pull_basic(op, a, t, s);
        case kPullHess: return launch_tiled_pull_hess(op, a, t, s);
        default: return launch_tiled_pull_dot(op, a, t, s);
    }
}

cudaError_t launch_push_tiled(int op, const LaunchArgs& a, const TileCfg& t, cudaStream_t s) {
    return op == kPush ? launch_tiled_push(op, a, t, s) : launch_tiled_push_grad(op, a, t, s);
}

TileGrid tile_grid(const LaunchArgs& a, const TileCfg& c) { return make_grid(a, c); }

namespace {
// One warp waits on an mbarrier that no copy or thread will ever complete, with
// a caller-given cycle limit: the bounded wait gives up, records the timeout in
// this unit's status word and the kernel returns normally.
__global__ void k_bounded_wait_probe(long long limit) {
    __shared__ __align__(8) unsigned long long bar;
    const unsigned a = smem_addr(&bar);
    if (threadIdx.x == 0) {
        mbar_init(a, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    mbar_wait_limit(a, 0u, limit);
    __syncwarp();
    if (threadIdx.x == 0) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(a) : "memory");
}
}  // namespace

cudaError_t launch_bounded_wait_probe(long long limit_cycles, cudaStream_t s) {
    k_bounded_wait_probe<<<1, 32, 0, s>>>(limit_cycles);
    return cudaGetLastError();
}

unsigned read_device_status(bool reset) {
    unsigned v = status_pull_basic(reset);
    v |= status_pull_hess(reset);
    v |= status_pull_dot(reset);
    v |= status_push(reset);
    v |= status_push_grad(reset);
    v |= status_fused(reset);
    v |= status_batch(reset);
    v |= status_ws_pull(reset);
    v |= status_ws_hess(reset);
    v |= status_ws_grad_dot(reset);
    v |= status_ws_hess_dot(reset);
    v |= status_push_affine(reset);
    v |= unit_status(reset);   // the bounded-wait probe of this unit
    return v;
}

}  // namespace pp
