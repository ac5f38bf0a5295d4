// C ABI of the sm_100a Fourier-slice operators: argument validation, geometry set-up,
// zero-fill of atomically accumulated outputs and kernel dispatch.  Declarations and the
// reference interfaces each entry point replaces are in include/b200proj.h.
#include "b200proj.h"

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <climits>
#include <cstdint>
#include <mutex>
#include <type_traits>

#include "brick_scatter.cuh"
#include "cell_scatter.cuh"

namespace {

using namespace b200proj;

thread_local char g_error[512] = "";

int fail(int code, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_error, sizeof(g_error), fmt, ap);
    va_end(ap);
    return code;
}

int cuda_fail(cudaError_t e, const char* what) {
    return fail(B200PROJ_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

struct Launch {
    SliceGeom g;
    dim3 grid;
    int64_t B, P;
    size_t rec_count;    // voxels in [B, (R,) R, Rh]
    size_t pix_count;    // pixels in [B, P, N, Nh]
};

// Validate the arguments common to all operators and derive the kernel geometry.
int prepare(Launch& L, int dim, int64_t B, int64_t R, int64_t B_rot, const void* rot,
            const void* shifts, int64_t B_shift, int64_t P, int64_t N, int interpolation,
            double oversampling, double cutoff) {
    g_error[0] = 0;
    if (interpolation != B200PROJ_LINEAR && interpolation != B200PROJ_CUBIC)
        return fail(B200PROJ_ERR_ARGUMENT, "Supported interpolation methods: 'linear', 'cubic'");
    if (B < 1 || P < 0) return fail(B200PROJ_ERR_ARGUMENT, "batch size must be >= 1 and pose count >= 0 (B=%lld, P=%lld)", (long long)B, (long long)P);
    if (N < 2 || (N % 2) != 0) return fail(B200PROJ_ERR_ARGUMENT, "projection boxsize (%lld) must be even and >= 2", (long long)N);
    if (R < 2 || (R % 2) != 0) return fail(B200PROJ_ERR_ARGUMENT, "reconstruction boxsize (%lld) must be even and >= 2", (long long)R);
    if (rot == nullptr) return fail(B200PROJ_ERR_ARGUMENT, "rotations pointer is NULL");
    if (B_rot != 1 && B_rot != B) return fail(B200PROJ_ERR_ARGUMENT, "Batch size of rotations must be 1 or same as reconstruction (B_rot=%lld, B=%lld)", (long long)B_rot, (long long)B);
    if (shifts != nullptr && B_shift != 1 && B_shift != B)
        return fail(B200PROJ_ERR_ARGUMENT, "Batch size of shifts must be 1 or same as reconstruction (B_shift=%lld, B=%lld)", (long long)B_shift, (long long)B);
    if (!(oversampling > 0.0) || !std::isfinite(oversampling))
        return fail(B200PROJ_ERR_ARGUMENT, "oversampling must be a positive finite number");
    if (std::isnan(cutoff)) return fail(B200PROJ_ERR_ARGUMENT, "fourier_radius_cutoff is NaN");
    if ((double)N * oversampling > 1073741824.0)
        return fail(B200PROJ_ERR_LIMIT, "N * oversampling = %g puts sample coordinates beyond 2^30", (double)N * oversampling);

    const int64_t Nh = N / 2 + 1, Rh = R / 2 + 1;
    const int64_t vol = (dim == 3 ? R : 1) * R * Rh;
    if (vol > INT_MAX) return fail(B200PROJ_ERR_LIMIT, "reconstruction of box %lld exceeds 2^31-1 voxels per batch item", (long long)R);
    if (N > 2048) return fail(B200PROJ_ERR_LIMIT, "projection boxsize %lld exceeds 2048", (long long)N);
    if (P * dim * dim > INT_MAX / 2) return fail(B200PROJ_ERR_LIMIT, "too many poses per batch item (%lld)", (long long)P);

    SliceGeom& g = L.g;
    g.N = (int)N; g.Nh = (int)Nh; g.R = (int)R; g.Rh = (int)Rh; g.half = (int)(R / 2);
    g.P = (int)P;
    g.tiles_j = (int)((Nh + kTileJ - 1) / kTileJ);
    g.tiles_i = (int)((N + kTileI - 1) / kTileI);
    g.rot_stride_b = (B_rot == 1) ? 0 : (int)(P * dim * dim);
    g.has_shift = shifts != nullptr;
    g.shift_stride_b = (!g.has_shift || B_shift == 1) ? 0 : (int)(P * 2);
    const float rc = (float)cutoff;
    g.cutoff_sq = rc * rc;
    g.cutoff_sq_d = cutoff * cutoff;
    g.os = oversampling;
    g.phase_scale = -2.0 * M_PI / (double)(float)N;
    g.n_f = (float)N;
    g.inv_n = (float)(1.0 / (double)N);
    g.phase_scale_f = (float)g.phase_scale;
    g.shift_scale = -2.0 * M_PI / (double)N;
    g.vol_elems = vol;
    g.order = nullptr;
    g.pack_index = nullptr;
    g.pack_count = 0;
    g.replicas = 1;
    g.replica_stride = 0;

    if (B * P > INT_MAX / 2) return fail(B200PROJ_ERR_LIMIT, "B*P = %lld slices exceed the grid limit; split the poses into chunks", (long long)(B * P));
    g.BP = (int)(B * P);
    g.slice_pixels = (int)(N * Nh);
    g.os_f = (float)oversampling;
    g.os_is_float = ((double)g.os_f == oversampling);
    g.sparse_samples = oversampling >= 1.5;
    // exact for tile < 2^16 whenever tiles_j <= 2^16 (the numbers of tiles per slice are far below)
    g.tiles_j_magic = g.tiles_j == 1 ? 0u : (unsigned)(((1ull << 32) + (unsigned long long)g.tiles_j - 1) / (unsigned long long)g.tiles_j);
    // x = tile, (y, z) = the slice (see block_work for the three decodings)
    unsigned gy, gz;
    if (B > 1 && P >= 1 && P <= 32768 && B <= 65535) {
        g.decode = 1;
        gy = (unsigned)P;
        gz = (unsigned)B;
    } else {
        g.decode = (B == 1) ? 0 : 2;
        const int64_t bp = B * P;
        gy = (unsigned)(bp < 32768 ? (bp > 0 ? bp : 1) : 32768);
        gz = (unsigned)((bp + 32767) / 32768 > 0 ? (bp + 32767) / 32768 : 1);
    }
    L.grid = dim3((unsigned)(g.tiles_j * g.tiles_i), gy, gz);
    L.B = B; L.P = P;
    L.rec_count = (size_t)B * (size_t)vol;
    L.pix_count = (size_t)B * (size_t)P * (size_t)N * (size_t)Nh;
    return B200PROJ_OK;
}

int check_launch(const char* what) {
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? B200PROJ_OK : cuda_fail(e, what);
}

int zero_async(void* p, size_t bytes, cudaStream_t s) {
    if (p == nullptr || bytes == 0) return B200PROJ_OK;
    const cudaError_t e = cudaMemsetAsync(p, 0, bytes, s);
    return e == cudaSuccess ? B200PROJ_OK : cuda_fail(e, "cudaMemsetAsync");
}

// Clear up to three outputs (NULL or empty: none).  What is below a few MB goes into one launch; a memset runs at
// full bandwidth but costs a launch per output.
int zero_outputs(cudaStream_t s, void* a, size_t na, void* b, size_t nb, void* c = nullptr, size_t nc = 0) {
    void* p[3] = {a, b, c};
    const size_t n[3] = {na, nb, nc};
    ZeroRegions z{};
    int small = 0;
    size_t words = 0;
    for (int r = 0; r < 3; ++r) {
        if (p[r] == nullptr || n[r] == 0) continue;
        if (n[r] > (4u << 20)) {
            if (int rc = zero_async(p[r], n[r], s)) return rc;
            continue;
        }
        z.p[small] = (unsigned*)p[r];
        z.n[small++] = n[r] / 4;
        words += n[r] / 4;
    }
    if (small == 0) return B200PROJ_OK;
    if (small == 1) return zero_async(z.p[0], z.n[0] * 4, s);
    const size_t blocks = (words + 1023) / 1024;
    zero_regions_kernel<<<(unsigned)(blocks < 1184 ? blocks : 1184), 256, 0, s>>>(z);
    return check_launch("zero_regions launch");
}

// Slab plan of the slab-ordered 3D back-projection: volumes whose planes of one batch item
// exceed 160 MB are processed in slabs of at most `slab_mb` MB of planes.  `eager` lowers the
// threshold to 120 MB: an interleaved accumulator (16 bytes per voxel) just above L2 (box 256:
// 135 MB) loses its sectors between hits when the samples are sparse (linear taps at oversampling
// >= 1.5: 4.4x the compulsory DRAM traffic in one pass), and two slab passes then cost less than
// that (11.2 -> 10.65 ms per 50,000 slices); with dense samples (oversampling 1) or cubic footprints
// the second visit of the pixels costs more than the evictions (measured 6 % and 1.5 % slower).
// Tunable for experiments through B200PROJ_SLAB_MB / B200PROJ_SLAB_MIN_MB /
// B200PROJ_SLAB_MIN_MB_EAGER (read once).
struct SlabPlan { int slabs, planes; };
SlabPlan slab_plan(int64_t R, bool has_weights, bool interleaved = false, bool eager = false) {
    static const double slab_mb = [] { const char* e = getenv("B200PROJ_SLAB_MB"); return e ? atof(e) : 64.0; }();
    static const double min_mb = [] { const char* e = getenv("B200PROJ_SLAB_MIN_MB"); return e ? atof(e) : 160.0; }();
    static const double min_mb_e = [] { const char* e = getenv("B200PROJ_SLAB_MIN_MB_EAGER"); return e ? atof(e) : 120.0; }();
    const double plane_bytes = (double)R * (double)(R / 2 + 1) * (interleaved ? 16.0 : has_weights ? 12.0 : 8.0);
    const double threshold = (eager && min_mb_e < min_mb) ? min_mb_e : min_mb;
    if (slab_mb <= 0.0 || plane_bytes * (double)R <= threshold * 1e6) return {1, (int)R};
    // 16-byte voxels: fewer, larger reductions per plane leave room for 1.4x the bytes (measured)
    int planes = (int)(slab_mb * (interleaved ? 1.4 : 1.0) * 1e6 / plane_bytes);
    if (planes < 1) planes = 1;
    const int slabs = (int)((R + planes - 1) / planes);
    return {slabs, planes};
}

// Copies of a small reconstruction or interleaved workspace over which the slices of one call are spread: reductions
// onto less than ~2 MB run at 55-60 % of the rate they reach on a larger target (probe: 146 instead
// of 254 G taps/s at 128 KB), so a reconstruction of `bytes` bytes gets the power of two of copies
// that brings it to 2 MiB, at most 32 and at most one per 32 slices.
int workspace_replicas(double bytes, int64_t P) {
    int r = 1;
    while (r < 32 && bytes * r < 2097152.0 && P >= 32 * (int64_t)(2 * r)) r *= 2;
    return r;
}

// Launch the slab-ordered kernel into an interleaved accumulator for slabs [first, first + count).
void launch_slab_interleaved(const Launch& L, cudaStream_t s, bool cubic, const float* proj, const float* weights,
                             const float* rot, const float* shifts, float4* acc, const SlabPlan& plan, int first, int count) {
    const dim3 grid((unsigned)(L.B * L.P), (unsigned)count, 1);
    if (cubic)
        backproject_slab_kernel<true, true, true><<<grid, kBlockThreads, 0, s>>>((const float2*)proj, weights, rot, shifts, nullptr, nullptr, acc, L.g, plan.planes, first);
    else
        backproject_slab_kernel<false, true, true><<<grid, kBlockThreads, 0, s>>>((const float2*)proj, weights, rot, shifts, nullptr, nullptr, acc, L.g, plan.planes, first);
}

// Linear forward projection with two pixels per lane (project_forw_rows2_kernel); B200PROJ_LINEAR_ROWS2=0
// selects the one-pixel kernel for comparisons (read once).
bool linear_rows2() {
    static const bool on = [] { const char* e = getenv("B200PROJ_LINEAR_ROWS2"); return e ? atoi(e) != 0 : true; }();
    return on;
}


// ---- brick-stationary kernels: plan and launch ---------------------------------------------------------
struct BrickLaunch {
    BrickPlan plan;
    int64_t bricks;          // of one batch item, for rotations
    size_t items;            // capacity of the item list
    size_t item_bytes, rec_bytes;
    size_t bytes;            // workspace
    int64_t slices;
    double pixels, in_ball;  // of the call: pixels inside the cutoff, bricks that can hold some
    bool forced, use;
};

// Pixels of a slice inside the cutoff.
double pixels_inside(int64_t N, double cutoff) {
    const double r = cutoff < 0.0 ? 0.0 : cutoff, n = (double)N / 2.0;
    const double all = (double)N * (double)(N / 2 + 1);
    if (r >= n * 1.4143) return all;
    const double disc = M_PI / 2.0 * r * r + r;
    return disc < all ? disc : all;
}

// Geometry and item list for bricks of D sample positions, `blocks` of them resident on the GPU.
template <typename D>
BrickLaunch brick_layout(int64_t B, int64_t P, int64_t N, double os, double cutoff, double blocks, double min_target, bool outside) {
    BrickLaunch L{};
    static const int force = [] { const char* e = getenv("B200PROJ_BRICKS"); return e ? atoi(e) : -1; }();   // 0 / 1: never / always, for tests
    if (force == 0 || os < 1.0 || !(cutoff >= 0.0) || P < 1) return L;
    if (force != 1 && (double)B * (double)P * (double)N * (double)(N / 2 + 1) < 6e5) return L;      // below all lines
    const double corner = sqrt((double)N * N / 2.0);
    const double reach = (cutoff < corner ? cutoff : corner) * os;
    if (reach > 1000.0) return L;
    const double pixels = pixels_inside(N, cutoff) * (double)B * (double)P;
    L.slices = B * P;
    L.plan.reach = (float)reach;
    L.plan.keep = 1 << 20;
    const int dims[3] = {D::x, D::y, D::z};
    // grid of a shell: that of the first with whole clusters of brick_setup_kernel around it, so that all lie on one lattice
    auto grid = [&](int shell, int* n) {
        const int span = 2 * ((int)ceil(reach * brick_stretch(shell)) + 2), inner = 2 * ((int)ceil(reach) + 2), cluster[3] = {8, 8, 4};
        int64_t cells = 1;
        for (int a = 0; a < 3; ++a) {
            n[a] = dims[a] ? (inner + dims[a] - 1) / dims[a] : 1;
            while (dims[a] && n[a] * dims[a] < span) n[a] += 2 * cluster[a];
            cells *= n[a];
        }
        return cells;
    };
    L.bricks = grid(0, L.plan.n);
    if (L.bricks * B > (1 << 26) || B * P > (1 << 26)) return L;
    L.plan.density = (float)(D::kDim == 3 ? (double)D::x * D::y * D::z / (4.0 * os * os) : (double)D::x * D::y / (2.0 * os * os));
    double target = pixels / (blocks * 8.0);
    if (target < min_target) target = min_target;
    L.plan.target = (float)target;
    L.plan.per_slice = (float)pixels_inside(N, cutoff);
    // the estimate counts bricks that stick out of the ball in full, and a few large ones may each count the whole slice
    L.plan.max_extra = (int)((L.bricks < 64 ? (double)L.bricks : 4.0) * pixels / target) + 64;
    static const int wait_ms = [] { const char* e = getenv("B200PROJ_BRICK_WAIT_MS"); return e ? atoi(e) : 10000; }();   // for tests
    L.plan.wait_ms = wait_ms < 0 ? 0 : wait_ms;
    // the shells' lists, as long as those beyond the first stay below 64 MB
    for (int l = 0; l < kShells; ++l) {
        int n[3];
        const double cells = (double)grid(l, n), r = reach * brick_stretch(l) + 1.0 + sqrt((double)dims[0] * dims[0] + (double)dims[1] * dims[1] + (double)dims[2] * dims[2]);
        const double round = D::kDim == 3 ? 4.19 * r * r * r / ((double)D::x * D::y * D::z) : M_PI * r * r / ((double)D::x * D::y);   // bricks that meet the ball lie in this one
        const size_t need = (size_t)((round < cells ? ceil(round) : cells) * (double)B) + (size_t)L.plan.max_extra;
        if (l > 0 && (L.items + need) * sizeof(int4) > (64u << 20)) break;
        for (int a = 0; a < 3; ++a) L.plan.n[a] = n[a];
        L.plan.at[l] = (int)L.items;
        L.plan.shells = l + 1;
        L.items += need;
    }
    for (int a = 0; a < 3; ++a) {
        L.plan.d[a] = dims[a];
        L.plan.lo[a] = -((L.plan.n[a] * dims[a]) / 2);
    }
    L.item_bytes = (L.items * sizeof(int4) + 255) & ~(size_t)255;
    L.rec_bytes = (size_t)(B * P) * (4 * sizeof(float4) + sizeof(float2));
    L.bytes = 256 + L.item_bytes + L.rec_bytes + (outside ? (size_t)(N * (N / 2 + 1)) * sizeof(int) : 0);
    L.pixels = pixels;
    L.in_ball = (D::kDim == 3 ? 4.19 * pow(reach + 12.0, 3) / ((double)D::x * D::y * D::z) : M_PI * pow(reach + 30.0, 2) / ((double)D::x * D::y)) * (double)B;
    L.forced = force == 1;
    L.use = true;
    return L;
}

// Forward projection: bricks pay once their pixels outweigh staging them, whatever their number, and a fixed cost
// (measured: 20 us and 26 ns per brick against 33 ps saved per cubic pixel at oversampling 2; dense samples are cheaper
// for the plain kernels, linear taps save only some 2 ps).
BrickLaunch gather_plan(int dim, int64_t B, int64_t P, int64_t N, bool cubic, bool records, double os, double cutoff) {
    if (dim == 2) {
        // cubic: measured crossings at 2-5 M pixels (27 M: 2.1-2.3x); linear taps are not faster at any size (0.6-1.05x)
        if (!cubic) return BrickLaunch{};
        BrickLaunch L = brick_layout<GatherBrick<2, true>>(B, P, N, os, cutoff, 148.0 * 3.0, 6000.0, true);
        L.use = L.use && (L.forced || L.pixels > 4.5e6);
        return L;
    }
    BrickLaunch L = cubic ? brick_layout<GatherBrick<3, true>>(B, P, N, os, cutoff, 148.0 * 3.0, 3000.0, true)
                          : brick_layout<GatherBrick<3, false>>(B, P, N, os, cutoff, 148.0 * 4.0, 3000.0, true);
    const double need = cubic ? (1.2e6 + 900.0 * L.in_ball) * (os < 2.0 ? 2.0 / os : 1.0)
                              : (10e6 + 3100.0 * L.in_ball) * (records ? 0.6 : 1.0);
    // linear taps: small volumes meet a slice in too few pixels per brick (box 38 oversampled twice: 1.8x slower)
    L.use = L.use && (L.forced || (L.pixels > need && (cubic || L.plan.reach > 84.f)));
    return L;
}

// Cubic scatter (below the sizes of pixel lists; linear taps: plain kernels, see brick_scatter.cuh).
template <int DIM, bool WEIGHTS>
BrickLaunch scatter_layout(int64_t B, int64_t P, int64_t N, double os, double cutoff) {
    using C = Scatter<DIM, WEIGHTS>;
    // 2D items are alike and flush many copies: a few per block are enough (8 per block: 5-20 % slower)
    return brick_layout<typename C::Brick>(B, P, N, os, cutoff, 148.0 * C::kBlocks * (DIM == 2 ? 0.4 : 1.0), 3000.0, false);
}
BrickLaunch scatter_plan(int dim, int64_t B, int64_t P, int64_t N, bool cubic, bool weights, double os, double cutoff) {
    if (!cubic) return BrickLaunch{};
    if (dim == 2) {
        BrickLaunch L = weights ? scatter_layout<2, true>(B, P, N, os, cutoff) : scatter_layout<2, false>(B, P, N, os, cutoff);
        // measured at 9 M pixels: weighted 1.3-1.4x, else 1.0-1.35x (dense samples 1.5x and more: the plain kernels contend); 27 M: 1.1-1.7x;
        // reconstructions that fill less than a tile gain nothing
        L.use = L.use && (L.forced || (L.pixels > (weights || os < 1.25 ? 4.5e6 : 9e6) && L.plan.reach > 24.f));
        return L;
    }
    BrickLaunch L = weights ? scatter_layout<3, true>(B, P, N, os, cutoff) : scatter_layout<3, false>(B, P, N, os, cutoff);
    // measured crossings with the plain kernels, in M pixels: 0.8 / 1.7 / 5 for box-128 / 256 / 400 gradients, 0.55 / 0.8 / 0.9 with weights
    L.use = L.use && (L.forced || L.pixels > (weights ? 0.6e6 + 45.0 * L.in_ball : 0.75e6 + 430.0 * L.in_ball));
    return L;
}

// Scratch a call can use: 16-byte aligned and, for the brick kernels, large enough.  What is not is left alone and the
// plain kernels run.
bool scratch_aligned(const void* workspace) { return workspace != nullptr && (reinterpret_cast<uintptr_t>(workspace) & 15u) == 0; }
bool runs_in(const BrickLaunch& L, const void* workspace, size_t workspace_bytes) {
    return L.use && scratch_aligned(workspace) && workspace_bytes >= L.bytes;
}

BrickWork brick_work(const BrickLaunch& L, void* workspace) {
    BrickWork w;
    w.header = (int*)workspace;
    w.items = (int4*)((char*)workspace + 256);
    w.recs = (float4*)((char*)workspace + 256 + L.item_bytes);
    w.shifts = (float2*)(w.recs + 4 * (size_t)L.slices);
    w.outside = (int*)((char*)workspace + 256 + L.item_bytes + L.rec_bytes);
    return w;
}

template <int DIM>
int brick_setup(const BrickLaunch& bl, const BrickWork& w, const Launch& L, const float* rot, const float* shifts, bool outside, cudaStream_t s, Gate gate = {}) {
    if (int rc = zero_async(w.header, 80, s)) return rc;
    const int64_t clusters = (int64_t)((bl.plan.n[0] + 7) / 8) * ((bl.plan.n[1] + 7) / 8) * ((bl.plan.n[2] + 3) / 4) * L.B;
    const int64_t slices = (L.B * L.P + 255) / 256;
    brick_setup_kernel<DIM><<<(unsigned)(1 + clusters + slices), 256, 0, s>>>(rot, shifts, w, L.g, bl.plan, (int)L.B, outside ? 1 : 0, gate);
    return check_launch("brick_setup launch");
}

template <int DIM, bool CUBIC, bool SAVE>
int launch_brick_forw(const Launch& L, const BrickLaunch& bl, void* workspace, const float* rec, const float* rot, const float* shifts,
                      float* out, float* derivs, cudaStream_t s) {
    const BrickWork w = brick_work(bl, workspace);
    if (int rc = brick_setup<DIM>(bl, w, L, rot, shifts, true, s)) return rc;
    constexpr size_t smem = sizeof(float2) * BrickShape<DIM, CUBIC>::kVoxels + sizeof(GatherBlock);
    const cudaError_t e = cudaFuncSetAttribute(brick_forw_kernel<DIM, CUBIC, SAVE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "brick_forw shared memory");
    brick_forw_kernel<DIM, CUBIC, SAVE><<<148 * (CUBIC ? 3 : 4), kBlockThreads, smem, s>>>((const float2*)rec, rot, shifts, (float2*)out, (float2*)derivs, w, L.g, bl.plan);
    return check_launch("brick_forw launch");
}

template <int DIM, bool WEIGHTS, bool DUP, bool INTERLEAVED = false>
int launch_brick_scatter(const Launch& L, const BrickLaunch& bl, void* workspace, const float* proj, const float* weights, const float* rot,
                         const float* shifts, float* vol, float* wvol, cudaStream_t s, float4* accum = nullptr, Gate gate = {}) {
    using C = Scatter<DIM, WEIGHTS>;
    const BrickWork w = brick_work(bl, workspace);
    BrickLaunch kept = bl;
    kept.plan.keep = L.g.half;
    if (int rc = brick_setup<DIM>(kept, w, L, rot, shifts, false, s, gate)) return rc;
    constexpr size_t smem = sizeof(typename C::Shared);
    static_assert((smem + 1024) * C::kBlocks <= 233472, "shared memory of an SM");
    const cudaError_t e = cudaFuncSetAttribute(brick_scatter_kernel<DIM, WEIGHTS, DUP, INTERLEAVED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "brick_scatter shared memory");
    brick_scatter_kernel<DIM, WEIGHTS, DUP, INTERLEAVED><<<148 * C::kBlocks, C::kThreads, smem, s>>>((const float2*)proj, weights, rot, shifts, (float2*)vol, wvol, accum, w, L.g, bl.plan, gate);
    return check_launch("brick_scatter launch");
}

// ---- pixel lists: plan and launch ---------------------------------------------------------------------------
struct ListLaunch {
    ListPlan plan;
    size_t count_bytes, item_bytes, pose_bytes, inside_bytes, block_bytes, bytes;
    int64_t slices;          // of the call
    double pixels;           // of the call
    bool forced, use;
};

// Pixels of a slice that a list holds, and an upper bound of their pairs (as list_setup_kernel finds them).
void listed_pixels(int64_t N, double cutoff, int64_t* pixels, int64_t* pairs) {
    const float rc = (float)cutoff;
    const double room = (double)(rc * rc);
    *pixels = *pairs = 0;
    for (int64_t kr = 1 - N / 2; kr <= N / 2; ++kr) {
        const double left = room - (double)(kr * kr);
        if (!(left >= 0.0)) continue;
        // the last column within the cutoff; a cutoff beyond the slice (infinite ones too) is cut to it first
        int64_t j = left >= (double)(N / 2) * (double)(N / 2) ? N / 2 : (int64_t)sqrt(left);
        while (j < N / 2 && (double)((j + 1) * (j + 1)) <= left) ++j;
        while ((double)(j * j) > left) --j;
        *pixels += j + 1;
        *pairs += j / 2 + 1;
        if (kr < 0 || kr == N / 2) --*pixels;             // the mirrored half of column 0
    }
}

// A grid of bricks over all samples with taps inside a reconstruction of box R.  `blocks` of the kernel fit the GPU.
ListLaunch list_layout(int dim, int64_t B, int64_t R, int64_t P, int64_t N, double os, double cutoff, double blocks) {
    ListLaunch L{};
    static const int force = [] { const char* e = getenv("B200PROJ_LISTS"); return e ? atoi(e) : -1; }();   // 0 / 1: never / always, for tests
    if (force == 0 || B < 1 || P < 1 || N < 2 || N > 2048 || R < 2 || R > 4096 || !(cutoff >= 0.0) || !(os > 0.0) || (double)(float)os != os) return L;
    const double rough = (double)B * (double)P * (double)N * (double)(N / 2 + 1);
    if (force != 1 && rough < 6e5) return L;                     // below all lines
    ListPlan& p = L.plan;
    const int log2[3] = {dim == 3 ? ListBrick<3>::kLogX : ListBrick<2>::kLogX, dim == 3 ? ListBrick<3>::kLogY : ListBrick<2>::kLogY, ListBrick<3>::kLogZ};
    const int64_t far = R / 2 + 2;                               // cells of samples with a tap inside lie below this, from -this on
    int64_t bricks = B;
    for (int a = 0; a < 3; ++a) {
        // a whole number of bricks on either side of 0 (of c: one)
        const int64_t size = (int64_t)1 << log2[a], above = (far + size - 1) / size, n = a == 0 ? above + 1 : a < dim ? 2 * above : 1;
        p.n[a] = (int)n;
        p.lo[a] = a == 0 ? (int)-size : a < dim ? (int)(-above * size) : 0;
        bricks *= n;
        while (((int64_t)1 << p.bits) < n) ++p.bits;
        p.fit[a] = (float)(above * size) - 0.5f;
        if (a > 0) p.round[a - 1] = kRound - (float)(p.lo[a] / size);
    }
    const double corner = sqrt((double)N * (double)N / 2.0);
    p.row_zero = 8388608.f + (float)(N / 2 - 1);
    p.reach = (float)((cutoff < corner ? cutoff : corner) * os * 1.00001);
    while (((int64_t)1 << p.bits_j) < N / 2 + 1) ++p.bits_j;
    while (((int64_t)1 << p.bits_i) < N) ++p.bits_i;
    int64_t inside, pairs;
    listed_pixels(N, cutoff, &inside, &pairs);
    if (bricks > (1 << 24) || (B << (dim * p.bits)) > (1 << 28) || B * P > (1 << 26) || inside < 1) return L;
    p.bricks = (int)bricks;
    p.item_bricks = (int)(bricks / B);
    p.inside = (int)inside;
    p.pairs = (int)pairs;
    L.slices = B * P;
    L.pixels = (double)inside * (double)L.slices;
    // slices of one pass over the list: at most 2^30 entries, and what the bits of an entry can name
    static const int64_t list_entries = [] { const char* e = getenv("B200PROJ_LIST_ENTRIES"); return e && atoll(e) > 0 ? (int64_t)atoll(e) : (int64_t)1 << 30; }();   // for tests
    const int64_t by_list = list_entries / inside > 1 ? list_entries / inside : 1, by_bits = (int64_t)1 << (32 - p.bits_i - p.bits_j < 26 ? 32 - p.bits_i - p.bits_j : 26);
    const int64_t most_slices = by_list < by_bits ? by_list : by_bits, passes = (L.slices + most_slices - 1) / most_slices;
    p.slices = (int)((L.slices + passes - 1) / passes);
    const int64_t entries = inside * p.slices;
    p.capacity = (unsigned)entries;
    const double most = (double)entries / (blocks * 8.0);
    p.most = most < 4096.0 ? 4096 : most > 8192.0 ? 8192 : (int)most;
    const size_t up = 255, items = (size_t)(bricks < entries ? bricks : entries) + (size_t)(entries / p.most) + 1;
    L.item_bytes = (items * sizeof(int4) + up) & ~up;
    L.pose_bytes = ((size_t)L.slices * 2 * sizeof(float4) + up) & ~up;
    L.inside_bytes = ((size_t)pairs * sizeof(unsigned) + up) & ~up;
    static const int shared = [] { const char* e = getenv("B200PROJ_LIST_SHARED"); return e ? atoi(e) : kListBricks; }();   // for tests
    if (p.item_bricks <= (shared < kListBricks ? shared : kListBricks) && B <= 65535) {
        // few bricks: counted in shared memory, a run of slices per block (some 16 blocks per SM)
        int64_t run = (p.slices + 148 * 16 - 1) / (148 * 16);
        p.run = (int)(run < 1 ? 1 : run);
        L.block_bytes = ((size_t)B * (size_t)((P + p.run - 1) / p.run) * (size_t)p.item_bricks * sizeof(unsigned) + up) & ~up;
        if (L.block_bytes > (64u << 20)) p.run = 0, L.block_bytes = 0;
    }
    // slices of a block that counts in global memory: several make a shorter grid, which a call whose lists are left aside waits for (0.5 ns a
    // block).  They follow one another, so that the lists keep the order of the slices (persistent blocks that took slices far apart: sums 5 % slower)
    const int64_t blocks_of = ((pairs + kListPairs - 1) / kListPairs) * p.slices;
    p.turn = blocks_of < 16384 ? 1 : 4;
    // counters of a brick (see list_pixels_kernel): half of the bricks of the grid meet slices
    for (p.subs = 1; p.run == 0 && p.subs < 8 && 2 * p.subs * bricks <= 80000;) p.subs *= 2;
    // their places: an odd factor near the golden ratio of the power of two of groups sends neighbours far apart
    unsigned groups = 1;
    while (8ll * groups < bricks) groups *= 2;
    p.groups = groups - 1;
    p.spread = (unsigned)(0.6180339887 * (double)groups) | 1u;
    L.count_bytes = ((size_t)groups * 8 * (size_t)p.subs * sizeof(unsigned) + up) & ~up;
    L.bytes = 256 + L.count_bytes + L.item_bytes + L.pose_bytes + L.inside_bytes + L.block_bytes + (size_t)entries * sizeof(unsigned);
    L.forced = force == 1;
    L.use = true;
    return L;
}

ListWork list_work(const ListLaunch& L, void* workspace) {
    ListWork w;
    char* at = (char*)workspace;
    w.header = (int*)at;
    w.count = (unsigned*)(at += 256);
    w.items = (int4*)(at += L.count_bytes);
    w.poses = (float4*)(at += L.item_bytes);
    w.inside = (unsigned*)(at += L.pose_bytes);
    w.block_count = (unsigned*)(at += L.inside_bytes);
    w.list = (unsigned*)(at += L.block_bytes);
    return w;
}

int copies_wanted(int dim, double one, int64_t B, int64_t P, int64_t N, bool cubic, bool pose_gradients);
// Scratch of the scatter that runs when the lists are left aside (see Gate).  weights: 1 to a volume of their own, 2 into 16-byte voxels.
size_t without_lists_bytes(int dim, int64_t B, int64_t R, int64_t P, int64_t N, bool cubic, int weights, double os, double cutoff) {
    const BrickLaunch bl = scatter_plan(dim, B, P, N, cubic, weights != 0, os, cutoff);
    if (bl.use) return bl.bytes;
    if (weights == 2 || (dim == 3 && slab_plan(R, weights != 0).slabs > 1)) return 0;
    const double one = (double)B * (dim == 3 ? R : 1) * R * (R / 2 + 1) * (double)(weights ? sizeof(float4) : sizeof(float2));
    const int copies = weights ? workspace_replicas(one, P) : copies_wanted(dim, one, B, P, N, cubic, false);
    return weights || copies > 1 ? (size_t)one * (size_t)copies : 0;
}
// When the lists are left aside: calls in which a brick's pixels share fewer than `crowd` of its cells (see list_setup_kernel; 128 lies between the
// 190 and more of poses that are spread and the 80 and less of those that are not), and only where the scatter without lists is then faster.
// Measured, without / from lists, weighted (unweighted): 3D linear, 10,000 slices of 128 x 65 oversampled twice: tilt series 1.46 / 1.58 (1.22 / 1.29) ms, in steps of
// 3 degrees 1.46 / 1.98 (1.22 / 1.56), one plane 1.39 / 1.41 (1.08 / 1.25), one pose 2.6 / 3.7 (2.1 / 2.8), ten poses 2.2 / 3.8, a hundred 2.2 / 2.3 (1.45 / 1.78), half of the
// slices in one plane 1.78 / 1.43 (1.27 / 1.25); 4,096 of 400 x 201 into volumes of their own: tilt series 7.3 / 7.5, in steps 7.4 / 10.1, one plane 8.9 / 5.3, ten poses 12.6 / 13.9;
// not oversampled 0.7-1.1x.  2D, all slices turned alike / not turned, oversampled twice, cubic: 4 M pixels 0.77 / 0.46x of the time from lists,
// 10 M 1.1 / 0.9x, 30 M and more 1.1-1.3x, but 64 x 33 references 0.85x at any number; linear: 22 M 1.0 / 0.79x, 45 M 1.2 / 0.85x, 51 M and
// more 1.0-1.5x / 0.95-1.05x.  3D cubic: 1.1-4x, except one pose and ten poses onto boxes of 64 and 96 (0.75-0.95x), which from here look like one plane (2x).
void list_crowd_rule(ListLaunch& L, int dim, int64_t B, int64_t R, int64_t P, int64_t N, bool cubic, int weights, double os, double cutoff) {
    static const float force = [] { const char* e = getenv("B200PROJ_LIST_CROWD"); return e ? (float)atof(e) : -1.f; }();   // number of cells, for tests
    const bool gains = dim == 3 ? !cubic : cubic ? L.pixels < 7e6 || R <= 72 : L.pixels < 5e7;
    L.plan.crowd = P < 2 || (dim == 3 && cubic) ? 0.f : force >= 0.f ? force : gains ? 128.f : 0.f;
    if (L.plan.crowd == 0.f) return;
    L.plan.probes = dim == 3 ? 256 : 64;
    const size_t other = 256 + without_lists_bytes(dim, B, R, P, N, cubic, weights, os, cutoff);
    if (other > L.bytes) L.bytes = other;
}
// Scatters from pixel lists: above a number of pixels that grows with the bricks (a brick costs its latency and its flush
// however few pixels it has).  Measured crossings with the kernels used otherwise (in M pixels; bricks inside the ball of the samples), with
// weights / without: 3D cubic, oversampled twice: 134 bricks 3 / 4, 1,072 2.3 / 3.5, 8,578 9 / 8, 68,600 55 / 50; not oversampled 0.5 / 0.8
// and 1 / 0.9 of 134 and 1,072.  3D linear 10 / 17, 8.5 / 14, 7 / 26, 36 / 40; 3 / 5, 4.3 / 7.  2D cubic, tiles: 6 1.8 / 3, 25 1.4 / 2.2, 100
// 1.4 / 2.3, 402 2.4 / 4.  2D linear 25 / 40, 10 / 35, 10.5 / 38, 25 / 50.  3D linear into 16-byte voxels, whose plain kernel reduces faster: 8,578 bricks 11, 68,600
// 51, 262,000 185.  Far above them 1.25-1.7x (3D), 1.2-1.7x (2D).  (Uniform poses; for others see list_crowd_rule.)  The pixels are those of one
// pass over the list: each pass clears, plans and flushes all bricks.
ListLaunch list_scatter_plan(int dim, int64_t B, int64_t R, int64_t P, int64_t N, bool cubic, int weights, double os, double cutoff) {
    ListLaunch L = list_layout(dim, B, R, P, N, os, cutoff, 148.0 * 4);
    if (!L.use) return L;
    list_crowd_rule(L, dim, B, R, P, N, cubic, weights, os, cutoff);
    if (L.forced) return L;
    const double r = L.plan.reach < (float)R * 0.5f ? L.plan.reach : (double)R * 0.5;
    const double bricks = (double)B * (dim == 3 ? 2.094 * r * r * r / 512.0 : 1.571 * r * r / 256.0);
    const bool dense = os < 1.25;
    double line;
    if (dim == 3) line = cubic ? (dense ? 0.9e6 : weights ? 2.5e6 : 3.2e6) + 750.0 * bricks
                               : (weights ? (dense ? 3.5e6 : 9e6) : (dense ? 6e6 : 16e6)) + (weights ? 400.0 : 800.0) * bricks;
    else line = cubic ? (weights ? 1.6e6 : 2.4e6) + 4e3 * bricks : (weights ? 11e6 : 36e6) + 3e4 * bricks + 2e8 / bricks;
    if (dim == 3 && !cubic && weights == 2 && !dense && line < 6e6 + 680.0 * bricks) line = 6e6 + 680.0 * bricks;
    return r > 24.0 && (double)L.plan.inside * (double)L.plan.slices > line ? L : ListLaunch{};
}
bool runs_in(const ListLaunch& L, const void* workspace, size_t workspace_bytes) {
    return L.use && scratch_aligned(workspace) && workspace_bytes >= L.bytes;
}

// For each pass over the list: sort the pixels, then run(work, plan).
template <int DIM, typename Run>
int with_lists(const Launch& L, const ListLaunch& ll, void* workspace, const float* rot, const float* shifts, cudaStream_t s, Run run) {
    const ListWork w = list_work(ll, workspace);
    ListPlan pl = ll.plan;
    const int per_pass = pl.slices;
    for (int64_t first = 0; first < ll.slices; first += per_pass) {
        pl.first = (int)first;
        pl.slices = (int)(ll.slices - first < per_pass ? ll.slices - first : per_pass);
        if (int rc = zero_async(w.header, 256 + ll.count_bytes, s)) return rc;
        const unsigned tiles = (unsigned)(L.g.tiles_i * ((L.g.Nh + 31) / 32));
        list_setup_kernel<DIM><<<tiles + (unsigned)((ll.slices + 255) / 256 + pl.probes), 256, 0, s>>>(rot, shifts, w, L.g, pl);
        if (int rc = check_launch("list_setup launch")) return rc;
        const unsigned across = (unsigned)((pl.pairs + kListPairs - 1) / kListPairs), down = (unsigned)((pl.slices + pl.turn - 1) / pl.turn);
        dim3 grid(across, down < 32768u ? down : 32768u, (down + 32767u) / 32768u);
        if (pl.run > 0) grid = dim3((unsigned)((L.P + pl.run - 1) / pl.run), (unsigned)L.B, 1);
        if (pl.run > 0) list_pixels_kernel<DIM, true, true><<<grid, 256, 0, s>>>(w, L.g, pl);
        else list_pixels_kernel<DIM, true, false><<<grid, 256, 0, s>>>(w, L.g, pl);
        if (int rc = check_launch("list_pixels (count) launch")) return rc;
        const int64_t places = L.B << (DIM * pl.bits);
        list_plan_kernel<DIM><<<(unsigned)((places + 255) / 256), 256, 0, s>>>(w, pl, (int)L.B);
        if (int rc = check_launch("list_plan launch")) return rc;
        if (pl.run > 0) list_pixels_kernel<DIM, false, true><<<grid, 256, 0, s>>>(w, L.g, pl);
        else list_pixels_kernel<DIM, false, false><<<grid, 256, 0, s>>>(w, L.g, pl);
        if (int rc = check_launch("list_pixels launch")) return rc;
        if (int rc = run(w, pl)) return rc;
    }
    return B200PROJ_OK;
}

template <int DIM, bool CUBIC, bool WEIGHTS, bool DUP, bool INTERLEAVED>
int run_list_scatter(const Launch& L, const ListLaunch& ll, void* workspace, const float* proj, const float* weights, const float* rot,
                     const float* shifts, float* vol, float* wvol, cudaStream_t s, float4* accum) {
    using C = std::conditional_t<DIM == 3 && CUBIC, CubicSums<WEIGHTS>, CellSums<DIM, CUBIC, WEIGHTS>>;
    constexpr size_t smem = sizeof(typename C::Shared);
    static_assert((smem + 1024) * C::kBlocks <= 233472, "shared memory of an SM");
    auto kernel = [] {
        if constexpr (DIM == 3 && CUBIC) return cell_cubic_sums_kernel<WEIGHTS, DUP, INTERLEAVED>;
        else return cell_sums_kernel<DIM, CUBIC, WEIGHTS, DUP, INTERLEAVED>;
    }();
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "cell_sums shared memory");
    const ScatterTarget<WEIGHTS, INTERLEAVED> to{(float2*)vol, wvol, accum};
    return with_lists<DIM>(L, ll, workspace, rot, shifts, s, [&](const ListWork& w, const ListPlan& pl) {
        kernel<<<148 * C::kBlocks, C::kThreads, smem, s>>>((const float2*)proj, weights, to, w, L.g, pl);
        if (int rc = check_launch("cell_sums launch")) return rc;
        scatter_rest_kernel<DIM, CUBIC, WEIGHTS, DUP><<<148 * 4, 256, 0, s>>>((const float2*)proj, weights, rot, shifts, to, w, L.g, pl);
        return check_launch("scatter_rest launch");
    });
}
template <int DIM, bool WEIGHTS, bool DUP, bool INTERLEAVED = false>
int launch_list_scatter(const Launch& L, const ListLaunch& ll, bool cubic, void* workspace, const float* proj, const float* weights, const float* rot,
                        const float* shifts, float* vol, float* wvol, cudaStream_t s, float4* accum = nullptr) {
    return cubic ? run_list_scatter<DIM, true, WEIGHTS, DUP, INTERLEAVED>(L, ll, workspace, proj, weights, rot, shifts, vol, wvol, s, accum)
                 : run_list_scatter<DIM, false, WEIGHTS, DUP, INTERLEAVED>(L, ll, workspace, proj, weights, rot, shifts, vol, wvol, s, accum);
}

// Copies of a small complex reconstruction (all batch items: `one` bytes) over which the slices of a scatter without
// weights are spread.  They cost a clear, a sum over the copies and two launches (3-5 us; small calls lose up to half), and
// gain where many reductions meet on few sectors.  In reductions per byte, measured on both sides of the lines: 2D, cubic /
// linear, 264 KB: 32 a byte 0.95 / 1.0x, 64 1.1 / 1.1x; 3D 461 KB cubic: 5 a byte 0.9x, 22 1.1x; 1.08 MB cubic: 10 0.95x, 32
// 1.1x; 1.5 MB cubic: 14 0.93x, 43 1.1x.  Linear reductions leave in pairs and gain nothing from 0.7 MB on (0.96-1.04x).  Beside
// the gather of the pose gradients they weigh less: linear 0.93-1.04x up to 80 a byte, 1.06x and more from 130 on; 2D
// cubic, 149-264 KB (of one batch item): 0.96x at 65, 1.0x at 300; below 0.1 MB 1.1x at 65.
int copies_wanted(int dim, double one, int64_t B, int64_t P, int64_t N, bool cubic, bool pose_gradients) {
    const int t = cubic ? 4 : 2;
    const double sums = (double)B * (double)P * (double)N * (double)(N / 2 + 1) * (dim == 3 ? t * t * t : t * t);
    double per_byte = dim == 3 && one <= 1.2e6 ? 15.0 : 36.0;
    if (pose_gradients && !cubic) per_byte = 120.0;
    else if (pose_gradients && dim == 2 && one > 1e5 * (double)B) per_byte = 250.0;
    if (sums < 1e6 || sums < per_byte * one || (!cubic && one > 5.5e5)) return 1;
    return workspace_replicas(one, P);
}
// As many of them as the workspace holds; sets the kernels' geometry.
int scatter_copies(Launch& L, int dim, bool cubic, bool pose_gradients, const void* workspace, size_t workspace_bytes) {
    if (!scratch_aligned(workspace)) return 1;
    const size_t one = L.rec_count * sizeof(float2);
    int copies = copies_wanted(dim, (double)one, L.B, L.P, L.g.N, cubic, pose_gradients);
    while (copies > 1 && (size_t)copies * one > workspace_bytes) copies /= 2;
    L.g.replicas = copies;
    L.g.replica_stride = copies > 1 ? (long long)L.rec_count : 0;
    return copies;
}
int add_copies(const Launch& L, const void* workspace, int copies, float* rec, cudaStream_t s, bool accumulate = false) {
    const size_t blocks = (L.rec_count + 255) / 256;
    add_copies_kernel<<<(unsigned)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, s>>>((const float2*)workspace, (float2*)rec, L.rec_count, copies, accumulate);
    return check_launch("add_copies launch");
}

// The scatter of a call whose lists are left aside (linear taps, and cubic ones in 2D): what runs calls without lists, behind a gate that is shut
// unless they are.  The outputs are cleared.  accum: 16-byte voxels instead of vol and wvol.
template <int DIM, bool WEIGHTS, bool DUP>
int scatter_without_lists(Launch L, const ListLaunch& ll, bool cubic, void* workspace, size_t workspace_bytes, const float* proj, const float* weights,
                          const float* rot, const float* shifts, float* vol, float* wvol, float4* accum, double os, double cutoff, bool accumulate, cudaStream_t s) {
    const Gate gate{(const int*)workspace, ll.plan.crowd};
    if (gate.crowd == 0.f) return B200PROJ_OK;
    void* scratch = (char*)workspace + 256;
    const size_t bytes = workspace_bytes - 256;
    const BrickLaunch bl = scatter_plan(DIM, L.B, L.P, L.g.N, cubic, WEIGHTS, os, cutoff);
    if (DIM == 2 && runs_in(bl, scratch, bytes)) return launch_brick_scatter<DIM, WEIGHTS, DUP>(L, bl, scratch, proj, weights, rot, shifts, vol, wvol, s, nullptr, gate);
    const float2* p = (const float2*)proj;
    auto zero = [&](size_t n) {
        gated_zero_kernel<<<148 * 8, 256, 0, s>>>((float4*)scratch, (n + 15) / 16, gate);
        return check_launch("gated_zero launch");
    };
    // slab passes: up to four slices to a block, as long as a slab that all slices lie in has some 2,000 blocks (2,048 slices of one plane, box 800: 4.74 ms,
    // with four to a block 5.0; idle blocks 0.06 ms of 6.4)
    const int per = L.g.BP < 4096 ? 1 : L.g.BP < 8192 ? 2 : 4;
    const unsigned by_slices = (unsigned)((L.g.BP + per - 1) / per);
    // several tiles to a block, as long as there are some ten blocks per place on the GPU
    const int64_t most = (int64_t)L.grid.x * L.g.BP / 8192;
    const int tiles = (int)(most < 1 ? 1 : most < (int64_t)L.grid.x ? most : L.grid.x);
    const dim3 grid((L.grid.x + tiles - 1) / tiles, L.grid.y, L.grid.z);
    if constexpr (WEIGHTS) {
        if constexpr (DIM == 3) {
            const SlabPlan apart = slab_plan(L.g.R, true);
            if (accum == nullptr && apart.slabs > 1) {
                gated_slab_kernel<true, false><<<dim3(by_slices, (unsigned)apart.slabs, 1), kBlockThreads, 0, s>>>(p, weights, rot, shifts, (float2*)vol, wvol, nullptr, L.g, apart.planes, per, gate);
                return check_launch("gated_slab launch");
            }
        }
        float4* to = accum;
        if (to == nullptr) {
            const size_t one = L.rec_count * sizeof(float4);
            L.g.replicas = workspace_replicas((double)one, L.P);
            while (L.g.replicas > 1 && (size_t)L.g.replicas * one > bytes) L.g.replicas /= 2;
            L.g.replica_stride = (long long)L.rec_count;
            to = (float4*)scratch;
            if (int rc = zero((size_t)L.g.replicas * one)) return rc;
        }
        const SlabPlan plan = DIM == 3 ? slab_plan(L.g.R, true, true, accum == nullptr && os >= 1.5) : SlabPlan{1, L.g.R};
        if (DIM == 3 && plan.slabs > 1)
            gated_slab_kernel<true, true><<<dim3(by_slices, (unsigned)plan.slabs, 1), kBlockThreads, 0, s>>>(p, weights, rot, shifts, nullptr, nullptr, to, L.g, plan.planes, per, gate);
        else if (DIM == 2 && cubic)
            gated_interleaved_kernel<2, true><<<grid, kBlockThreads, 0, s>>>(p, weights, rot, shifts, to, L.g, tiles, gate);
        else
            gated_interleaved_kernel<DIM, false><<<grid, kBlockThreads, 0, s>>>(p, weights, rot, shifts, to, L.g, tiles, gate);
        if (int rc = check_launch("gated scatter launch")) return rc;
        if (accum != nullptr) return B200PROJ_OK;
        fold_interleaved_kernel<<<148 * 16, 256, 0, s>>>(to, (float2*)vol, wvol, L.rec_count, accumulate ? 1 : 0, L.g.replicas, L.rec_count, gate);
        return check_launch("fold_interleaved launch");
    } else {
        if constexpr (DIM == 3 && DUP) {
            const SlabPlan plan = slab_plan(L.g.R, false);
            if (plan.slabs > 1) {
                gated_slab_kernel<false, false><<<dim3(by_slices, (unsigned)plan.slabs, 1), kBlockThreads, 0, s>>>(p, nullptr, rot, shifts, (float2*)vol, nullptr, nullptr, L.g, plan.planes, per, gate);
                return check_launch("gated_slab launch");
            }
        }
        const int copies = scatter_copies(L, DIM, cubic, false, scratch, bytes);
        if (copies > 1)
            if (int rc = zero((size_t)copies * L.rec_count * sizeof(float2))) return rc;
        float2* to = copies > 1 ? (float2*)scratch : (float2*)vol;
        if (DIM == 2 && cubic) gated_scatter_kernel<2, true, DUP><<<grid, kBlockThreads, 0, s>>>(p, rot, shifts, to, L.g, tiles, gate);
        else gated_scatter_kernel<DIM, false, DUP><<<grid, kBlockThreads, 0, s>>>(p, rot, shifts, to, L.g, tiles, gate);
        if (int rc = check_launch("gated scatter launch")) return rc;
        if (copies == 1) return B200PROJ_OK;
        add_copies_kernel<<<148 * 16, 256, 0, s>>>((const float2*)scratch, (float2*)vol, L.rec_count, copies, accumulate, gate);
        return check_launch("add_copies launch");
    }
}

// Of the sizes of scratch that a call has a use for, the larger one that is at most `most` bytes.
size_t largest_within(size_t most, size_t a, size_t b) {
    if (a > most) a = 0;
    if (b > most) b = 0;
    return a > b ? a : b;
}
// A scatter from lists and, behind the gate, the one without.
template <int DIM, bool WEIGHTS, bool DUP>
int scatter_by_lists(const Launch& L, const ListLaunch& ll, bool cubic, void* workspace, size_t workspace_bytes, const float* proj, const float* weights,
                     const float* rot, const float* shifts, float* vol, float* wvol, float4* accum, double os, double cutoff, bool accumulate, cudaStream_t s) {
    int rc;
    if constexpr (DIM == 3 && WEIGHTS) {
        rc = accum != nullptr ? launch_list_scatter<3, true, true, true>(L, ll, cubic, workspace, proj, weights, rot, shifts, nullptr, nullptr, s, accum)
                              : launch_list_scatter<3, true, true>(L, ll, cubic, workspace, proj, weights, rot, shifts, vol, wvol, s);
    } else {
        rc = launch_list_scatter<DIM, WEIGHTS, DUP>(L, ll, cubic, workspace, proj, weights, rot, shifts, vol, wvol, s);
    }
    return rc ? rc : scatter_without_lists<DIM, WEIGHTS, DUP>(L, ll, cubic, workspace, workspace_bytes, proj, weights, rot, shifts, vol, wvol, accum, os, cutoff, accumulate, s);
}

// ---- operator bodies, templated on the dimensionality and the real type (float | double) ------------------------------------
template <int DIM, typename Real>
int project_forw(const Real* rec, int64_t B, int64_t R, const Real* rot, int64_t B_rot,
                 const Real* shifts, int64_t B_shift, int64_t P, int64_t N, int interpolation,
                 double os, double cutoff, Real* out, const int32_t* pose_order, void* stream,
                 void* workspace = nullptr, size_t workspace_bytes = 0) {
    Launch L;
    if (int rc = prepare(L, DIM, B, R, B_rot, rot, shifts, B_shift, P, N, interpolation, os, cutoff)) return rc;
    if (rec == nullptr || out == nullptr) return fail(B200PROJ_ERR_ARGUMENT, "reconstruction / output pointer is NULL");
    L.g.order = pose_order;
    if (P == 0) return B200PROJ_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if constexpr (std::is_same<Real, float>::value) {
        const BrickLaunch bl = workspace != nullptr ? gather_plan(DIM, B, P, N, interpolation == B200PROJ_CUBIC, false, os, cutoff) : BrickLaunch{};
        if (runs_in(bl, workspace, workspace_bytes)) {
            if (interpolation == B200PROJ_CUBIC) return launch_brick_forw<DIM, true, false>(L, bl, workspace, rec, rot, shifts, out, nullptr, s);
            if constexpr (DIM == 3) return launch_brick_forw<3, false, false>(L, bl, workspace, rec, rot, shifts, out, nullptr, s);
        }
    }
    const C2<Real>* v = (const C2<Real>*)rec;
    C2<Real>* o = (C2<Real>*)out;
    if (interpolation == B200PROJ_CUBIC) {
        project_forw_kernel<DIM, true><<<L.grid, kBlockThreads, 0, s>>>(v, rot, shifts, o, L.g);
    } else if (linear_rows2()) {
        // linear: two pixels per lane, a block covers 16 columns x 32 rows
        const dim3 grid((unsigned)(L.g.tiles_j * ((N + 2 * kTileI - 1) / (2 * kTileI))), L.grid.y, L.grid.z);
        project_forw_rows2_kernel<DIM><<<grid, kBlockThreads, 0, s>>>(v, rot, shifts, o, L.g);
    } else {
        project_forw_kernel<DIM, false><<<L.grid, kBlockThreads, 0, s>>>(v, rot, shifts, o, L.g);
    }
    return check_launch("project_forw launch");
}

template <int DIM, bool CUBIC, typename Real>
void launch_project_back(const Launch& L, cudaStream_t s, const C2<Real>* gp, const C2<Real>* rec,
                         const Real* rot, const Real* shifts, C2<Real>* grad_rec, Real* grad_rot,
                         Real* grad_shift) {
    const bool nr = grad_rot != nullptr, ns = grad_shift != nullptr;
#define B200PROJ_PB(NR, NS) \
    project_back_kernel<DIM, CUBIC, NR, NS><<<L.grid, kBlockThreads, 0, s>>>(gp, rec, rot, shifts, grad_rec, grad_rot, grad_shift, L.g)
    if (nr && ns) B200PROJ_PB(true, true);
    else if (nr) B200PROJ_PB(true, false);
    else if (ns) B200PROJ_PB(false, true);
    else B200PROJ_PB(false, false);
#undef B200PROJ_PB
}

template <int DIM, bool CUBIC, bool RECORDS>
void launch_project_back_saved(const Launch& L, cudaStream_t s, const float2* gp, const float2* out, const float2* derivs,
                               const float* rot, const float* shifts, float2* grad_rec, float* grad_rot, float* grad_shift) {
    const bool nr = grad_rot != nullptr, ns = grad_shift != nullptr;
#define B200PROJ_PBS(NR, NS) \
    project_back_saved_kernel<DIM, CUBIC, NR, NS, RECORDS><<<L.grid, kBlockThreads, 0, s>>>(gp, out, derivs, rot, shifts, grad_rec, grad_rot, grad_shift, L.g)
    if (nr && ns) B200PROJ_PBS(true, true);
    else if (nr) B200PROJ_PBS(true, false);
    else if (ns) B200PROJ_PBS(false, true);
    else B200PROJ_PBS(false, false);
#undef B200PROJ_PBS
}

template <int DIM, bool RECORDS>
void launch_pose_grad_saved(const Launch& L, cudaStream_t s, const float2* gp, const float2* out, const float2* derivs, float* grad_rot, float* grad_shift) {
    // one block per slice once that fills the GPU (8 blocks per SM), else the slice in parts of at least 1,024 pixels
    const int64_t fill = 148 * 8 / (int64_t)L.g.BP, most = (L.g.slice_pixels + 1023) / 1024;
    const dim3 grid((unsigned)L.g.BP, (unsigned)(fill < 1 ? 1 : fill < most ? fill : most), 1);
    if (grad_rot != nullptr && grad_shift != nullptr) pose_grad_saved_kernel<DIM, true, true, RECORDS><<<grid, kBlockThreads, 0, s>>>(gp, out, derivs, grad_rot, grad_shift, L.g);
    else if (grad_rot != nullptr) pose_grad_saved_kernel<DIM, true, false, RECORDS><<<grid, kBlockThreads, 0, s>>>(gp, out, derivs, grad_rot, grad_shift, L.g);
    else pose_grad_saved_kernel<DIM, false, true, RECORDS><<<grid, kBlockThreads, 0, s>>>(gp, out, derivs, grad_rot, grad_shift, L.g);
}

// Forward projection that also writes the pixels' derivatives (as planes, or as one record per pixel), and the
// backward pass from them (fp32).
template <int DIM, bool RECORDS = false>
int project_forw_saving(const float* rec, int64_t B, int64_t R, const float* rot, int64_t B_rot, const float* shifts,
                        int64_t B_shift, int64_t P, int64_t N, int interpolation, double os, double cutoff,
                        float* out, float* derivatives, const int32_t* pose_order, void* stream,
                        void* workspace = nullptr, size_t workspace_bytes = 0) {
    Launch L;
    if (int rc = prepare(L, DIM, B, R, B_rot, rot, shifts, B_shift, P, N, interpolation, os, cutoff)) return rc;
    if (rec == nullptr || out == nullptr || derivatives == nullptr) return fail(B200PROJ_ERR_ARGUMENT, "reconstruction / output / derivatives pointer is NULL");
    L.g.order = pose_order;
    if (P == 0) return B200PROJ_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (RECORDS && (reinterpret_cast<uintptr_t>(derivatives) & 31u) != 0) return fail(B200PROJ_ERR_ARGUMENT, "records must be 32-byte aligned");
    if constexpr (RECORDS || DIM == 2) {
        const BrickLaunch bl = workspace != nullptr ? gather_plan(DIM, B, P, N, interpolation == B200PROJ_CUBIC, true, os, cutoff) : BrickLaunch{};
        if (runs_in(bl, workspace, workspace_bytes)) {
            if (interpolation == B200PROJ_CUBIC) return launch_brick_forw<DIM, true, true>(L, bl, workspace, rec, rot, shifts, out, derivatives, s);
            if constexpr (DIM == 3) return launch_brick_forw<3, false, true>(L, bl, workspace, rec, rot, shifts, out, derivatives, s);
        }
    }
    if (interpolation == B200PROJ_CUBIC)
        project_forw_saving_kernel<DIM, true, RECORDS><<<L.grid, kBlockThreads, 0, s>>>((const float2*)rec, rot, shifts, (float2*)out, (float2*)derivatives, L.g);
    else
        project_forw_saving_kernel<DIM, false, RECORDS><<<L.grid, kBlockThreads, 0, s>>>((const float2*)rec, rot, shifts, (float2*)out, (float2*)derivatives, L.g);
    return check_launch("project_forw (saving derivatives) launch");
}

template <int DIM, bool RECORDS = false>
int project_back_saved(const float* grad_proj, const float* out, const float* derivatives, int64_t B, int64_t R,
                       const float* rot, int64_t B_rot, const float* shifts, int64_t B_shift, int64_t P, int64_t N,
                       int interpolation, double os, double cutoff, float* grad_rec, float* grad_rot, float* grad_shifts,
                       const int32_t* pose_order, void* stream, void* workspace = nullptr, size_t workspace_bytes = 0) {
    Launch L;
    if (int rc = prepare(L, DIM, B, R, B_rot, rot, shifts, B_shift, P, N, interpolation, os, cutoff)) return rc;
    L.g.order = pose_order;
    if (grad_proj == nullptr) return fail(B200PROJ_ERR_ARGUMENT, "grad_projections pointer is NULL");
    if (grad_rot != nullptr && derivatives == nullptr) return fail(B200PROJ_ERR_ARGUMENT, "grad_rotations requested but no saved derivatives given");
    if (grad_shifts != nullptr && (shifts == nullptr || out == nullptr))
        return fail(B200PROJ_ERR_ARGUMENT, "grad_shifts requested but no shifts / saved projections given");
    if (RECORDS && (reinterpret_cast<uintptr_t>(derivatives) & 15u) != 0) return fail(B200PROJ_ERR_ARGUMENT, "records must be 16-byte aligned");
    if (grad_rec == nullptr && grad_rot == nullptr && grad_shifts == nullptr) return B200PROJ_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const bool cubic = interpolation == B200PROJ_CUBIC;
    BrickLaunch bl{};
    ListLaunch ll{};
    if ((RECORDS || DIM == 2) && P > 0 && grad_rec != nullptr && workspace != nullptr) {
        // (linear: the kernel below, which forms the pose gradients on its way, is as fast where lists are left aside for it)
        if (cubic) ll = list_scatter_plan(DIM, B, R, P, N, cubic, 0, os, cutoff);
        ll.use = runs_in(ll, workspace, workspace_bytes);
        if (!ll.use) bl = scatter_plan(DIM, B, P, N, cubic, false, os, cutoff);
    }
    bl.use = runs_in(bl, workspace, workspace_bytes);
    const int copies = P > 0 && grad_rec != nullptr && !bl.use && !ll.use ? scatter_copies(L, DIM, cubic, false, workspace, workspace_bytes) : 1;
    if (int rc = zero_outputs(s, copies > 1 ? nullptr : grad_rec, L.rec_count * sizeof(float2), grad_rot, (size_t)B_rot * P * DIM * DIM * sizeof(float),
                              grad_shifts, (size_t)(shifts ? B_shift : 0) * P * 2 * sizeof(float))) return rc;
    if (P == 0) return B200PROJ_OK;
    const float2* gp = (const float2*)grad_proj;
    const float2* o = RECORDS && out == derivatives ? nullptr : (const float2*)out;      // the records themselves: their fourth entries
    const float2* d = (const float2*)derivatives;
    if (bl.use || ll.use) {
        // large scatter: brick by brick, the pose gradients in a streaming pass of their own
        if (int rc = ll.use ? scatter_by_lists<DIM, false, false>(L, ll, cubic, workspace, workspace_bytes, grad_proj, nullptr, rot, shifts, grad_rec, nullptr, nullptr, os, cutoff, false, s)
                            : launch_brick_scatter<DIM, false, false>(L, bl, workspace, grad_proj, nullptr, rot, shifts, grad_rec, nullptr, s)) return rc;
        if (grad_rot == nullptr && grad_shifts == nullptr) return B200PROJ_OK;
        grad_rec = nullptr;
    }
    if (grad_rec != nullptr) {
        if (copies > 1)
            if (int rc = zero_async(workspace, (size_t)copies * L.rec_count * sizeof(float2), s)) return rc;
        float2* to = copies > 1 ? (float2*)workspace : (float2*)grad_rec;
        if (cubic) launch_project_back_saved<DIM, true, RECORDS>(L, s, gp, o, d, rot, shifts, to, grad_rot, grad_shifts);
        else launch_project_back_saved<DIM, false, RECORDS>(L, s, gp, o, d, rot, shifts, to, grad_rot, grad_shifts);
        if (int rc = check_launch("project_back (saved derivatives) launch")) return rc;
        return copies > 1 ? add_copies(L, workspace, copies, grad_rec, s) : B200PROJ_OK;
    }
    launch_pose_grad_saved<DIM, RECORDS>(L, s, gp, o, d, grad_rot, grad_shifts);
    return check_launch("project_back (saved derivatives) launch");
}

template <int DIM, typename Real>
int project_back(const Real* grad_proj, const Real* rec, int64_t B, int64_t R, const Real* rot,
                 int64_t B_rot, const Real* shifts, int64_t B_shift, int64_t P, int64_t N,
                 int interpolation, double os, double cutoff, Real* grad_rec, Real* grad_rot,
                 Real* grad_shifts, const int32_t* pose_order, void* stream, void* workspace = nullptr, size_t workspace_bytes = 0) {
    Launch L;
    if (int rc = prepare(L, DIM, B, R, B_rot, rot, shifts, B_shift, P, N, interpolation, os, cutoff)) return rc;
    L.g.order = pose_order;
    if (grad_proj == nullptr || rec == nullptr || grad_rec == nullptr)
        return fail(B200PROJ_ERR_ARGUMENT, "grad_projections / reconstruction / grad_reconstruction pointer is NULL");
    if (grad_shifts != nullptr && shifts == nullptr)
        return fail(B200PROJ_ERR_ARGUMENT, "grad_shifts requested but no shifts given");
    cudaStream_t s = (cudaStream_t)stream;
    BrickLaunch bl{};
    ListLaunch ll{};
    if (std::is_same<Real, float>::value && P > 0 && grad_rot == nullptr && grad_shifts == nullptr && workspace != nullptr) {
        ll = list_scatter_plan(DIM, B, R, P, N, interpolation == B200PROJ_CUBIC, 0, os, cutoff);
        ll.use = runs_in(ll, workspace, workspace_bytes);
        if (!ll.use) bl = scatter_plan(DIM, B, P, N, interpolation == B200PROJ_CUBIC, false, os, cutoff);
    }
    bl.use = runs_in(bl, workspace, workspace_bytes);
    const int copies = P > 0 && std::is_same<Real, float>::value && !bl.use && !ll.use ? scatter_copies(L, DIM, interpolation == B200PROJ_CUBIC, grad_rot != nullptr || grad_shifts != nullptr, workspace, workspace_bytes) : 1;
    if (int rc = zero_outputs(s, copies > 1 ? nullptr : grad_rec, L.rec_count * sizeof(C2<Real>), grad_rot, (size_t)B_rot * P * DIM * DIM * sizeof(Real),
                              grad_shifts, (size_t)(shifts ? B_shift : 0) * P * 2 * sizeof(Real))) return rc;
    if (P == 0) return B200PROJ_OK;
    if constexpr (std::is_same<Real, float>::value) {
        if (ll.use) return scatter_by_lists<DIM, false, false>(L, ll, interpolation == B200PROJ_CUBIC, workspace, workspace_bytes, grad_proj, nullptr, rot, shifts, grad_rec, nullptr, nullptr, os, cutoff, false, s);
        if (bl.use) return launch_brick_scatter<DIM, false, false>(L, bl, workspace, grad_proj, nullptr, rot, shifts, grad_rec, nullptr, s);
    }
    if (copies > 1)
        if (int rc = zero_async(workspace, (size_t)copies * L.rec_count * sizeof(float2), s)) return rc;
    C2<Real>* to = copies > 1 ? (C2<Real>*)workspace : (C2<Real>*)grad_rec;
    if (interpolation == B200PROJ_CUBIC)
        launch_project_back<DIM, true>(L, s, (const C2<Real>*)grad_proj, (const C2<Real>*)rec, rot, shifts, to, grad_rot, grad_shifts);
    else
        launch_project_back<DIM, false>(L, s, (const C2<Real>*)grad_proj, (const C2<Real>*)rec, rot, shifts, to, grad_rot, grad_shifts);
    if (int rc = check_launch("project_back launch")) return rc;
    return copies > 1 ? add_copies(L, workspace, copies, (float*)grad_rec, s) : B200PROJ_OK;
}

template <int DIM, typename Real>
int backproject_forw(const Real* proj, const Real* weights, int64_t B, int64_t R,
                     const Real* rot, int64_t B_rot, const Real* shifts, int64_t B_shift,
                     int64_t P, int64_t N, int interpolation, double os, double cutoff,
                     Real* data_rec, Real* weight_rec, int accumulate, void* workspace,
                     size_t workspace_bytes, void* stream) {
    Launch L;
    if (int rc = prepare(L, DIM, B, R, B_rot, rot, shifts, B_shift, P, N, interpolation, os, cutoff)) return rc;
    if (proj == nullptr || data_rec == nullptr) return fail(B200PROJ_ERR_ARGUMENT, "projections / data_reconstruction pointer is NULL");
    if ((weights != nullptr) != (weight_rec != nullptr))
        return fail(B200PROJ_ERR_ARGUMENT, "weights and weight_reconstruction must be given together");
    if (R != b200proj_rec_boxsize(N, os))
        return fail(B200PROJ_ERR_ARGUMENT, "reconstruction boxsize %lld does not match ceil(N*oversampling) rounded up to even = %lld",
                    (long long)R, (long long)b200proj_rec_boxsize(N, os));
    cudaStream_t s = (cudaStream_t)stream;
    const bool cubic = interpolation == B200PROJ_CUBIC, hw = weights != nullptr;
    // Interleaved path: data and weight of a voxel share one 16-byte slot of the workspace
    // (one v4 reduction per tap), folded into the outputs afterwards.
    const size_t ws_one = L.rec_count * sizeof(float4);
    if constexpr (std::is_same<Real, float>::value) {
        const ListLaunch ll = P > 0 && workspace != nullptr ? list_scatter_plan(DIM, B, R, P, N, cubic, hw ? 1 : 0, os, cutoff) : ListLaunch{};
        if (runs_in(ll, workspace, workspace_bytes)) {
            if (!accumulate) {
                if (int rc = zero_outputs(s, data_rec, L.rec_count * sizeof(C2<Real>), weight_rec, L.rec_count * sizeof(Real))) return rc;
            }
            return hw ? scatter_by_lists<DIM, true, true>(L, ll, cubic, workspace, workspace_bytes, proj, weights, rot, shifts, data_rec, weight_rec, nullptr, os, cutoff, accumulate != 0, s)
                      : scatter_by_lists<DIM, false, true>(L, ll, cubic, workspace, workspace_bytes, proj, nullptr, rot, shifts, data_rec, nullptr, nullptr, os, cutoff, accumulate != 0, s);
        }
        const BrickLaunch bl = P > 0 && workspace != nullptr ? scatter_plan(DIM, B, P, N, cubic, hw, os, cutoff) : BrickLaunch{};
        if (runs_in(bl, workspace, workspace_bytes)) {
            if (!accumulate) {
                if (int rc = zero_outputs(s, data_rec, L.rec_count * sizeof(C2<Real>), weight_rec, L.rec_count * sizeof(Real))) return rc;
            }
            return hw ? launch_brick_scatter<DIM, true, true>(L, bl, workspace, proj, weights, rot, shifts, data_rec, weight_rec, s)
                      : launch_brick_scatter<DIM, false, true>(L, bl, workspace, proj, nullptr, rot, shifts, data_rec, nullptr, s);
        }
    }
    constexpr bool kIsF32 = std::is_same<Real, float>::value;  // workspace and slab paths exist in fp32 only
    if constexpr (kIsF32) {
    if (hw && P > 0 && !(DIM == 3 && slab_plan(R, hw).slabs > 1) && scratch_aligned(workspace) && workspace_bytes >= ws_one) {
        // small reconstructions: as many copies as the rule wants and the workspace holds
        int replicas = workspace_replicas((double)ws_one, P);
        while (replicas > 1 && (size_t)replicas * ws_one > workspace_bytes) replicas /= 2;
        L.g.replicas = replicas;
        L.g.replica_stride = (long long)L.rec_count;
        const size_t ws_need = (size_t)replicas * ws_one;
        if (int rc = zero_async(workspace, ws_need, s)) return rc;
        float4* acc = (float4*)workspace;
        const SlabPlan plan_i = (DIM == 3) ? slab_plan(R, true, true, /*eager=*/!cubic && os >= 1.5) : SlabPlan{1, (int)R};
        if (DIM == 3 && plan_i.slabs > 1)      // the 16-byte volume itself is beyond L2: slab-ordered passes
            launch_slab_interleaved(L, s, cubic, (const float*)proj, (const float*)weights, (const float*)rot, (const float*)shifts, acc, plan_i, 0, plan_i.slabs);
        else if (cubic)
            backproject_forw_interleaved_kernel<DIM, true><<<L.grid, kBlockThreads, 0, s>>>((const C2<Real>*)proj, weights, rot, shifts, acc, L.g);
        else
            backproject_forw_interleaved_kernel<DIM, false><<<L.grid, kBlockThreads, 0, s>>>((const C2<Real>*)proj, weights, rot, shifts, acc, L.g);
        if (int rc = check_launch("backproject_forw (interleaved) launch")) return rc;
        const size_t blocks = (L.rec_count + 255) / 256;
        fold_interleaved_kernel<<<(unsigned)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, s>>>(acc, (C2<Real>*)data_rec, weight_rec, L.rec_count, accumulate != 0,
                                                                                              replicas, L.rec_count);
        return check_launch("fold_interleaved launch");
    }
    }
    if constexpr (kIsF32) {
        // a small reconstruction without weights: copies of it in the workspace
        const int copies = !hw && P > 0 ? scatter_copies(L, DIM, cubic, false, workspace, workspace_bytes) : 1;
        if (copies > 1) {
            if (int rc = zero_async(workspace, (size_t)copies * L.rec_count * sizeof(float2), s)) return rc;
            if (cubic) backproject_forw_kernel<DIM, true, false><<<L.grid, kBlockThreads, 0, s>>>((const float2*)proj, weights, rot, shifts, (float2*)workspace, weight_rec, L.g);
            else backproject_forw_kernel<DIM, false, false><<<L.grid, kBlockThreads, 0, s>>>((const float2*)proj, weights, rot, shifts, (float2*)workspace, weight_rec, L.g);
            if (int rc = check_launch("backproject_forw (copies) launch")) return rc;
            return add_copies(L, workspace, copies, data_rec, s, accumulate != 0);
        }
    }
    if (!accumulate) {
        if (int rc = zero_outputs(s, data_rec, L.rec_count * sizeof(C2<Real>), weight_rec, L.rec_count * sizeof(Real))) return rc;
    }
    if (P == 0) return B200PROJ_OK;
    const C2<Real>* p = (const C2<Real>*)proj;
    C2<Real>* d = (C2<Real>*)data_rec;
    if constexpr (DIM == 3 && kIsF32) {
        // volumes beyond L2: slab-ordered passes that keep the active planes L2-resident
        const SlabPlan plan = slab_plan(R, hw);
        if (plan.slabs > 1) {
            const dim3 grid((unsigned)(B * P), (unsigned)plan.slabs, 1);
#define B200PROJ_SL(C, W) \
    backproject_slab_kernel<C, W><<<grid, kBlockThreads, 0, s>>>(p, weights, rot, shifts, d, weight_rec, nullptr, L.g, plan.planes, 0)
            if (cubic && hw) B200PROJ_SL(true, true);
            else if (cubic) B200PROJ_SL(true, false);
            else if (hw) B200PROJ_SL(false, true);
            else B200PROJ_SL(false, false);
#undef B200PROJ_SL
            return check_launch("backproject_forw (slab-ordered) launch");
        }
    }
#define B200PROJ_BP(C, W) \
    backproject_forw_kernel<DIM, C, W><<<L.grid, kBlockThreads, 0, s>>>(p, weights, rot, shifts, d, weight_rec, L.g)
    if (cubic && hw) B200PROJ_BP(true, true);
    else if (cubic) B200PROJ_BP(true, false);
    else if (hw) B200PROJ_BP(false, true);
    else B200PROJ_BP(false, false);
#undef B200PROJ_BP
    return check_launch("backproject_forw launch");
}

template <int DIM, bool CUBIC, typename Real>
void launch_backproject_back(const Launch& L, cudaStream_t s, const C2<Real>* gd, const Real* gw,
                             const C2<Real>* proj, const Real* rot, const Real* shifts,
                             C2<Real>* grad_proj, Real* grad_weights, Real* grad_rot,
                             Real* grad_shift) {
    const bool nr = grad_rot != nullptr, ns = grad_shift != nullptr;
    if constexpr (!CUBIC) {
        // enough slices and pixels: patches; the measurements stand at backproject_back_patches_kernel
        const int64_t patches = (int64_t)((L.g.N + 3) / 4) * ((L.g.Nh + 7) / 8);
        if (L.g.BP >= 2 * 148 && L.g.BP * patches >= 6000 && (sizeof(Real) == 4 || patches >= 64) && (nr || ns)) {
            // eight blocks per SM, and at most 16 patches a warp: what a block has left at the end is short, and few slices are under way at once
            const int64_t most = (patches + 7) / 8, fill = (148 * 8 + L.g.BP - 1) / L.g.BP, blocks = fill < most ? fill : most, least = (most + 15) / 16;
            const dim3 grid((unsigned)(blocks > least ? blocks : least), L.grid.y, L.grid.z);
#define B200PROJ_BB(NR, NS) \
    backproject_back_patches_kernel<DIM, NR, NS><<<grid, kBlockThreads, 0, s>>>(gd, gw, proj, rot, shifts, grad_proj, grad_weights, grad_rot, grad_shift, L.g)
            if (nr && ns) B200PROJ_BB(true, true);
            else if (nr) B200PROJ_BB(true, false);
            else B200PROJ_BB(false, true);
#undef B200PROJ_BB
            return;
        }
    }
#define B200PROJ_BB(NR, NS) \
    backproject_back_kernel<DIM, CUBIC, NR, NS><<<L.grid, kBlockThreads, 0, s>>>(gd, gw, proj, rot, shifts, grad_proj, grad_weights, grad_rot, grad_shift, L.g)
    if (nr && ns) B200PROJ_BB(true, true);
    else if (nr) B200PROJ_BB(true, false);
    else if (ns) B200PROJ_BB(false, true);
    else B200PROJ_BB(false, false);
#undef B200PROJ_BB
}

template <int DIM, typename Real>
int backproject_back(const Real* grad_data_rec, const Real* grad_weight_rec, const Real* proj,
                     int64_t B, int64_t R, const Real* rot, int64_t B_rot, const Real* shifts,
                     int64_t B_shift, int64_t P, int64_t N, int interpolation, double os,
                     double cutoff, Real* grad_proj, Real* grad_weights, Real* grad_rot,
                     Real* grad_shifts, const int32_t* pose_order, void* stream) {
    Launch L;
    if (int rc = prepare(L, DIM, B, R, B_rot, rot, shifts, B_shift, P, N, interpolation, os, cutoff)) return rc;
    L.g.order = pose_order;
    if (grad_data_rec == nullptr || grad_proj == nullptr)
        return fail(B200PROJ_ERR_ARGUMENT, "grad_data_rec / grad_projections pointer is NULL");
    if ((grad_rot != nullptr || grad_shifts != nullptr) && proj == nullptr)
        return fail(B200PROJ_ERR_ARGUMENT, "projections are needed for rotation / shift gradients");
    if (grad_shifts != nullptr && shifts == nullptr)
        return fail(B200PROJ_ERR_ARGUMENT, "grad_shifts requested but no shifts given");
    if (R != b200proj_rec_boxsize(N, os))
        return fail(B200PROJ_ERR_ARGUMENT, "grad_data_rec boxsize %lld does not match ceil(N*oversampling) rounded up to even = %lld",
                    (long long)R, (long long)b200proj_rec_boxsize(N, os));
    cudaStream_t s = (cudaStream_t)stream;
    if (int rc = zero_outputs(s, grad_rot, (size_t)B_rot * P * DIM * DIM * sizeof(Real), grad_shifts, (size_t)(shifts ? B_shift : 0) * P * 2 * sizeof(Real))) return rc;
    if (grad_weights != nullptr && grad_weight_rec == nullptr)   // weights given, no incoming gradient: zeros
        if (int rc = zero_async(grad_weights, L.pix_count * sizeof(Real), s)) return rc;
    if (P == 0) return B200PROJ_OK;
    if (interpolation == B200PROJ_CUBIC)
        launch_backproject_back<DIM, true>(L, s, (const C2<Real>*)grad_data_rec, grad_weight_rec, (const C2<Real>*)proj, rot, shifts, (C2<Real>*)grad_proj, grad_weights, grad_rot, grad_shifts);
    else
        launch_backproject_back<DIM, false>(L, s, (const C2<Real>*)grad_data_rec, grad_weight_rec, (const C2<Real>*)proj, rot, shifts, (C2<Real>*)grad_proj, grad_weights, grad_rot, grad_shifts);
    return check_launch("backproject_back launch");
}

// Weighted 3D back-projection that ADDS into a persistent interleaved accumulator (16-byte
// (re, im, w, 0) voxels): one v4 reduction per tap, nothing zero-filled or folded per call.
int backproject_accumulate(const float* proj, const float* weights, int64_t B, int64_t R, const float* rot,
                           int64_t B_rot, const float* shifts, int64_t B_shift, int64_t P, int64_t N,
                           int interpolation, double os, double cutoff, void* accumulator,
                           int slab_first, int slab_count, void* stream, void* workspace = nullptr, size_t workspace_bytes = 0) {
    Launch L;
    if (int rc = prepare(L, 3, B, R, B_rot, rot, shifts, B_shift, P, N, interpolation, os, cutoff)) return rc;
    if (proj == nullptr || weights == nullptr || accumulator == nullptr)
        return fail(B200PROJ_ERR_ARGUMENT, "projections, weights and accumulator are all required");
    if ((reinterpret_cast<uintptr_t>(accumulator) & 15u) != 0)
        return fail(B200PROJ_ERR_ARGUMENT, "accumulator must be 16-byte aligned");
    if (R != b200proj_rec_boxsize(N, os))
        return fail(B200PROJ_ERR_ARGUMENT, "reconstruction boxsize %lld does not match ceil(N*oversampling) rounded up to even = %lld",
                    (long long)R, (long long)b200proj_rec_boxsize(N, os));
    const SlabPlan plan = slab_plan(R, true, true);
    if (slab_count < 0) { slab_first = 0; slab_count = plan.slabs; }         // all slabs
    if (slab_first < 0 || slab_count < 1 || slab_first + slab_count > plan.slabs)
        return fail(B200PROJ_ERR_ARGUMENT, "slabs [%d, %d) outside the plan of %d slabs", slab_first, slab_first + slab_count, plan.slabs);
    if (P == 0) return B200PROJ_OK;
    cudaStream_t s = (cudaStream_t)stream;
    float4* acc = (float4*)accumulator;
    const bool cubic = interpolation == B200PROJ_CUBIC;
    if (workspace != nullptr && slab_count == plan.slabs) {
        const ListLaunch ll = list_scatter_plan(3, B, R, P, N, cubic, 2, os, cutoff);
        if (runs_in(ll, workspace, workspace_bytes)) return scatter_by_lists<3, true, true>(L, ll, cubic, workspace, workspace_bytes, proj, weights, rot, shifts, nullptr, nullptr, acc, os, cutoff, true, s);
        const BrickLaunch bl = scatter_plan(3, B, P, N, cubic, true, os, cutoff);
        if (runs_in(bl, workspace, workspace_bytes)) return launch_brick_scatter<3, true, true, true>(L, bl, workspace, proj, weights, rot, shifts, nullptr, nullptr, s, acc);
    }
    if (plan.slabs > 1) {
        launch_slab_interleaved(L, s, cubic, proj, weights, rot, shifts, acc, plan, slab_first, slab_count);
        return check_launch("backproject_accumulate (slab-ordered) launch");
    }
    if (cubic)
        backproject_forw_interleaved_kernel<3, true><<<L.grid, kBlockThreads, 0, s>>>((const float2*)proj, weights, rot, shifts, acc, L.g);
    else
        backproject_forw_interleaved_kernel<3, false><<<L.grid, kBlockThreads, 0, s>>>((const float2*)proj, weights, rot, shifts, acc, L.g);
    return check_launch("backproject_accumulate launch");
}

// pad + fftshift (pad != 0) or ifftshift + crop (pad == 0) of `batch` real arrays with `dims` axes.
template <typename Real>
int pad_shift(const Real* in, int64_t batch, int dims, int64_t n, int64_t m, int pad, Real* out, void* stream) {
    g_error[0] = 0;
    if (in == nullptr || out == nullptr) return fail(B200PROJ_ERR_ARGUMENT, "input / output pointer is NULL");
    if (dims != 2 && dims != 3) return fail(B200PROJ_ERR_ARGUMENT, "dims must be 2 or 3");
    if (batch < 1 || n < 1 || m < n || (m % 2) != 0)
        return fail(B200PROJ_ERR_ARGUMENT, "need batch >= 1, 1 <= n <= m and an even padded box (batch=%lld, n=%lld, m=%lld)", (long long)batch, (long long)n, (long long)m);
    const int64_t out_box = pad ? m : n;
    if (m > 8192 || batch * (dims == 3 ? out_box : 1) > 65535 * 32768ll || out_box > 65535)
        return fail(B200PROJ_ERR_LIMIT, "box %lld / batch %lld beyond what one launch indexes", (long long)m, (long long)batch);
    const int64_t gz = batch * (dims == 3 ? out_box : 1);
    if (gz > 65535) return fail(B200PROJ_ERR_LIMIT, "batch * box = %lld exceeds the grid limit; split the batch", (long long)gz);
    const dim3 grid((unsigned)((out_box + 255) / 256), (unsigned)((out_box + 3) / 4), (unsigned)gz), block(64, 4, 1);
    cudaStream_t s = (cudaStream_t)stream;
    const int lo = (int)((m - n) / 2);
    // 16-byte stores when every output row starts on a 16-byte boundary
    const bool vec = (out_box % 4) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
#define B200PROJ_PS(D, P, V) pad_shift_kernel<D, P, V><<<grid, block, 0, s>>>(in, out, (int)n, (int)m, lo, (int)batch)
    if (dims == 3) {
        if (pad) { if (vec) B200PROJ_PS(3, true, true); else B200PROJ_PS(3, true, false); }
        else     { if (vec) B200PROJ_PS(3, false, true); else B200PROJ_PS(3, false, false); }
    } else {
        if (pad) { if (vec) B200PROJ_PS(2, true, true); else B200PROJ_PS(2, true, false); }
        else     { if (vec) B200PROJ_PS(2, false, true); else B200PROJ_PS(2, false, false); }
    }
#undef B200PROJ_PS
    return check_launch("pad_shift launch");
}

template <typename Real>
int pose_order_3d(const Real* rot, int64_t B, int64_t B_rot, int64_t P, int32_t* order, void* stream) {
    g_error[0] = 0;
    if (rot == nullptr || order == nullptr) return fail(B200PROJ_ERR_ARGUMENT, "rotations / order pointer is NULL");
    if (B < 1 || P < 0) return fail(B200PROJ_ERR_ARGUMENT, "batch size must be >= 1 and pose count >= 0 (B=%lld, P=%lld)", (long long)B, (long long)P);
    if (B_rot != 1 && B_rot != B) return fail(B200PROJ_ERR_ARGUMENT, "Batch size of rotations must be 1 or same as reconstruction (B_rot=%lld, B=%lld)", (long long)B_rot, (long long)B);
    if (B * P > INT_MAX / 2 || B > 65535 * 32768ll) return fail(B200PROJ_ERR_LIMIT, "B*P = %lld slices exceed the grid limit; split the poses into chunks", (long long)(B * P));
    if (P == 0) return B200PROJ_OK;
    pose_order_kernel<<<(unsigned)B, kOrderBins, 0, (cudaStream_t)stream>>>(rot, B_rot == 1 ? 0ll : (long long)P * 9, (int)P, order);
    return check_launch("pose_order launch");
}

// ---- built-in scratch of the allocation-free back-projection entry point -----------------
// The array lives in every GPU context that loads this library, from load until exit.
constexpr long long kNoAllocMaxVoxels = B200PROJ_NOALLOC_MAX_VOXELS;
static __device__ __align__(256) float4 g_noalloc_accum[kNoAllocMaxVoxels];

constexpr int kNoAllocMaxDevices = 64;
float4* g_noalloc_ptr[kNoAllocMaxDevices] = {};
std::mutex g_noalloc_mutex;

// Device address of the built-in scratch on the CURRENT device.  In host code the array's
// name is only a stand-in; the address a kernel can use comes from cudaGetSymbolAddress,
// asked once per device with that device current.
int noalloc_scratch(float4** out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    if (dev < 0 || dev >= kNoAllocMaxDevices)
        return fail(B200PROJ_ERR_LIMIT, "device ordinal %d is beyond the %d devices the allocation-free entry point tracks", dev, kNoAllocMaxDevices);
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (g_noalloc_ptr[dev] == nullptr) {
        float4* ptr = nullptr;
        e = cudaGetSymbolAddress((void**)&ptr, g_noalloc_accum);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress");
        g_noalloc_ptr[dev] = ptr;
    }
    *out = g_noalloc_ptr[dev];
    return B200PROJ_OK;
}

}  // namespace

extern "C" {

int b200proj_version(void) { return 300; }

#ifndef B200PROJ_SOURCE_STAMP
#define B200PROJ_SOURCE_STAMP ""
#endif
const char* b200proj_source_stamp(void) { return B200PROJ_SOURCE_STAMP; }

const char* b200proj_last_error(void) { return g_error; }

size_t b200proj_backproject_workspace_bytes(int dim, int64_t B, int64_t R, int64_t P, int64_t N,
                                           int interpolation, int has_weights) {
    if ((dim != 2 && dim != 3) || B < 1 || R < 2 || P < 1 || N < 2) return 0;
    const double voxels = (double)B * (dim == 3 ? R : 1) * R * (R / 2 + 1);
    const int t = interpolation == B200PROJ_CUBIC ? 4 : 2;
    const double taps = (double)B * P * N * (N / 2 + 1) * (dim == 3 ? t * t * t : t * t);
    // worth it once the scatter outweighs the two extra passes over the volume
    if (taps < 4.0 * voxels) return 0;
    if (dim == 3 && slab_plan(R, has_weights != 0).slabs > 1) return 0;      // beyond-L2 volumes take the slab-ordered path
    const double one = voxels * (double)(has_weights ? sizeof(float4) : sizeof(float2));
    const int copies = has_weights ? workspace_replicas(one, P) : copies_wanted(dim, one, B, P, N, interpolation == B200PROJ_CUBIC, false);   // small reconstructions: several copies
    return has_weights || copies > 1 ? (size_t)one * (size_t)copies : 0;
}

int64_t b200proj_rec_boxsize(int64_t N, double oversampling) {
    const int64_t raw = (int64_t)std::ceil((double)N * oversampling);
    return raw + (raw % 2);
}

int b200proj_debug_index(int which, int R, int coordinate, int mirrored_in, int* mirrored_out) {
    SliceGeom g{};
    g.R = R; g.Rh = R / 2 + 1; g.half = R / 2;
    bool m = mirrored_in != 0;
    int r = INT_MIN;
    switch (which) {
        case 0: r = gather_col<false>(g, coordinate, m); break;
        case 1: r = gather_col<true>(g, coordinate, m); break;
        case 2: r = gather_line<false>(g, coordinate, m); break;
        case 3: r = gather_line<true>(g, coordinate, m); break;
        case 4: r = scatter_col(g, coordinate, m); break;
        case 5: r = scatter_line(g, coordinate, m); break;
        default: break;
    }
    if (mirrored_out != nullptr) *mirrored_out = m ? 1 : 0;
    return r;
}

int b200proj_project_2d_forw(const float* rec, int64_t B, int64_t R, const float* rot, int64_t B_rot,
                             const float* shifts, int64_t B_shift, int64_t P, int64_t N,
                             int interpolation, double oversampling, double cutoff, float* out,
                             void* stream) {
    return project_forw<2>(rec, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, out, nullptr, stream);
}
int b200proj_project_3d_to_2d_forw(const float* rec, int64_t B, int64_t R, const float* rot,
                                   int64_t B_rot, const float* shifts, int64_t B_shift, int64_t P,
                                   int64_t N, int interpolation, double oversampling, double cutoff,
                                   float* out, const int32_t* pose_order, void* stream) {
    return project_forw<3>(rec, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, out, pose_order, stream);
}

size_t b200proj_scatter_workspace_bytes_within(int dim, int64_t B, int64_t P, int64_t N, int interpolation, int has_weights, double oversampling, double cutoff, size_t most) {
    if (dim != 2 && dim != 3) return 0;
    const BrickLaunch bl = scatter_plan(dim, B, P, N, interpolation == B200PROJ_CUBIC, has_weights != 0, oversampling, cutoff);
    const ListLaunch ll = list_scatter_plan(dim, B, b200proj_rec_boxsize(N, oversampling), P, N, interpolation == B200PROJ_CUBIC, has_weights, oversampling, cutoff);
    return largest_within(most, ll.use ? ll.bytes : 0, bl.use ? bl.bytes : 0);
}
size_t b200proj_scatter_workspace_bytes(int dim, int64_t B, int64_t P, int64_t N, int interpolation, int has_weights, double oversampling, double cutoff) {
    return b200proj_scatter_workspace_bytes_within(dim, B, P, N, interpolation, has_weights, oversampling, cutoff, SIZE_MAX);
}
size_t b200proj_gradient_workspace_bytes_within(int dim, int64_t B, int64_t R, int64_t P, int64_t N, int interpolation, int pose_gradients,
                                                double oversampling, double cutoff, size_t most) {
    if ((dim != 2 && dim != 3) || B < 1 || R < 2 || P < 1 || N < 2) return 0;
    const bool cubic = interpolation == B200PROJ_CUBIC;
    if (pose_gradients == 0 || (pose_gradients == 2 && cubic)) {
        const ListLaunch ll = list_scatter_plan(dim, B, R, P, N, cubic, 0, oversampling, cutoff);
        const BrickLaunch bl = scatter_plan(dim, B, P, N, cubic, false, oversampling, cutoff);
        if (const size_t bytes = largest_within(most, ll.use ? ll.bytes : 0, bl.use ? bl.bytes : 0)) return bytes;
    }
    const double one = (double)B * (dim == 3 ? R : 1) * R * (R / 2 + 1) * (double)sizeof(float2);
    const int copies = copies_wanted(dim, one, B, P, N, cubic, pose_gradients == 1);
    return copies > 1 ? largest_within(most, (size_t)one * (size_t)copies, 0) : 0;
}
size_t b200proj_gradient_workspace_bytes(int dim, int64_t B, int64_t R, int64_t P, int64_t N, int interpolation, int pose_gradients,
                                         double oversampling, double cutoff) {
    return b200proj_gradient_workspace_bytes_within(dim, B, R, P, N, interpolation, pose_gradients, oversampling, cutoff, SIZE_MAX);
}
size_t b200proj_project_workspace_bytes(int dim, int64_t B, int64_t P, int64_t N, int interpolation, int records, double oversampling, double cutoff) {
    if (dim != 2 && dim != 3) return 0;
    const BrickLaunch bl = gather_plan(dim, B, P, N, interpolation == B200PROJ_CUBIC, records != 0, oversampling, cutoff);
    return bl.use ? bl.bytes : 0;
}
int b200proj_project_2d_forw_ws(const float* rec, int64_t B, int64_t R, const float* rot,
                                int64_t B_rot, const float* shifts, int64_t B_shift, int64_t P,
                                int64_t N, int interpolation, double oversampling, double cutoff,
                                float* out, void* workspace, size_t workspace_bytes, void* stream) {
    return project_forw<2>(rec, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, out, nullptr, stream, workspace, workspace_bytes);
}
int b200proj_project_2d_forw_saving_ws(const float* rec, int64_t B, int64_t R, const float* rot,
                                       int64_t B_rot, const float* shifts, int64_t B_shift, int64_t P,
                                       int64_t N, int interpolation, double oversampling, double cutoff,
                                       float* out, float* derivatives, void* workspace, size_t workspace_bytes, void* stream) {
    return project_forw_saving<2>(rec, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, out, derivatives, nullptr, stream, workspace, workspace_bytes);
}
int b200proj_project_3d_to_2d_forw_ws(const float* rec, int64_t B, int64_t R, const float* rot,
                                      int64_t B_rot, const float* shifts, int64_t B_shift, int64_t P,
                                      int64_t N, int interpolation, double oversampling, double cutoff,
                                      float* out, const int32_t* pose_order, void* workspace, size_t workspace_bytes, void* stream) {
    return project_forw<3>(rec, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, out, pose_order, stream, workspace, workspace_bytes);
}
int b200proj_project_3d_to_2d_forw_records(const float* rec, int64_t B, int64_t R, const float* rot,
                                           int64_t B_rot, const float* shifts, int64_t B_shift, int64_t P,
                                           int64_t N, int interpolation, double oversampling, double cutoff, float* out,
                                           float* records, const int32_t* pose_order, void* workspace, size_t workspace_bytes, void* stream) {
    return project_forw_saving<3, true>(rec, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, out, records, pose_order, stream, workspace, workspace_bytes);
}
int b200proj_project_3d_to_2d_back_records(const float* grad_proj, const float* out, const float* records,
                                           int64_t B, int64_t R, const float* rot, int64_t B_rot,
                                           const float* shifts, int64_t B_shift, int64_t P, int64_t N,
                                           int interpolation, double oversampling, double cutoff,
                                           float* grad_rec, float* grad_rot, float* grad_shifts,
                                           const int32_t* pose_order, void* workspace, size_t workspace_bytes, void* stream) {
    return project_back_saved<3, true>(grad_proj, out, records, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, grad_rec, grad_rot, grad_shifts, pose_order, stream, workspace, workspace_bytes);
}

int b200proj_project_2d_back(const float* grad_proj, const float* rec, int64_t B, int64_t R,
                             const float* rot, int64_t B_rot, const float* shifts, int64_t B_shift,
                             int64_t P, int64_t N, int interpolation, double oversampling,
                             double cutoff, float* grad_rec, float* grad_rot, float* grad_shifts,
                             void* stream) {
    return project_back<2>(grad_proj, rec, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, grad_rec, grad_rot, grad_shifts, nullptr, stream);
}
int b200proj_project_3d_to_2d_back(const float* grad_proj, const float* rec, int64_t B, int64_t R,
                                   const float* rot, int64_t B_rot, const float* shifts,
                                   int64_t B_shift, int64_t P, int64_t N, int interpolation,
                                   double oversampling, double cutoff, float* grad_rec,
                                   float* grad_rot, float* grad_shifts, const int32_t* pose_order,
                                   void* stream) {
    return project_back<3>(grad_proj, rec, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, grad_rec, grad_rot, grad_shifts, pose_order, stream);
}

int b200proj_project_2d_back_ws(const float* grad_proj, const float* rec, int64_t B, int64_t R,
                                const float* rot, int64_t B_rot, const float* shifts, int64_t B_shift, int64_t P, int64_t N,
                                int interpolation, double oversampling, double cutoff, float* grad_rec,
                                float* grad_rot, float* grad_shifts, void* workspace, size_t workspace_bytes, void* stream) {
    return project_back<2>(grad_proj, rec, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, grad_rec, grad_rot, grad_shifts, nullptr, stream, workspace, workspace_bytes);
}
int b200proj_project_2d_back_saved_ws(const float* grad_proj, const float* out, const float* derivatives,
                                      int64_t B, int64_t R, const float* rot, int64_t B_rot,
                                      const float* shifts, int64_t B_shift, int64_t P, int64_t N,
                                      int interpolation, double oversampling, double cutoff, float* grad_rec,
                                      float* grad_rot, float* grad_shifts, void* workspace, size_t workspace_bytes, void* stream) {
    return project_back_saved<2>(grad_proj, out, derivatives, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, grad_rec, grad_rot, grad_shifts, nullptr, stream, workspace, workspace_bytes);
}
int b200proj_project_3d_to_2d_back_ws(const float* grad_proj, const float* rec, int64_t B, int64_t R,
                                      const float* rot, int64_t B_rot, const float* shifts,
                                      int64_t B_shift, int64_t P, int64_t N, int interpolation,
                                      double oversampling, double cutoff, float* grad_rec,
                                      float* grad_rot, float* grad_shifts, const int32_t* pose_order,
                                      void* workspace, size_t workspace_bytes, void* stream) {
    return project_back<3>(grad_proj, rec, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, grad_rec, grad_rot, grad_shifts, pose_order, stream, workspace, workspace_bytes);
}

int b200proj_project_2d_forw_saving(const float* rec, int64_t B, int64_t R, const float* rot,
                                    int64_t B_rot, const float* shifts, int64_t B_shift, int64_t P,
                                    int64_t N, int interpolation, double oversampling, double cutoff,
                                    float* out, float* derivatives, void* stream) {
    return project_forw_saving<2>(rec, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, out, derivatives, nullptr, stream);
}
int b200proj_project_3d_to_2d_forw_saving(const float* rec, int64_t B, int64_t R, const float* rot,
                                          int64_t B_rot, const float* shifts, int64_t B_shift, int64_t P,
                                          int64_t N, int interpolation, double oversampling, double cutoff,
                                          float* out, float* derivatives, const int32_t* pose_order, void* stream) {
    return project_forw_saving<3>(rec, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, out, derivatives, pose_order, stream);
}
int b200proj_project_2d_back_saved(const float* grad_proj, const float* out, const float* derivatives,
                                   int64_t B, int64_t R, const float* rot, int64_t B_rot,
                                   const float* shifts, int64_t B_shift, int64_t P, int64_t N,
                                   int interpolation, double oversampling, double cutoff,
                                   float* grad_rec, float* grad_rot, float* grad_shifts, void* stream) {
    return project_back_saved<2>(grad_proj, out, derivatives, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, grad_rec, grad_rot, grad_shifts, nullptr, stream);
}
int b200proj_project_3d_to_2d_back_saved(const float* grad_proj, const float* out, const float* derivatives,
                                         int64_t B, int64_t R, const float* rot, int64_t B_rot,
                                         const float* shifts, int64_t B_shift, int64_t P, int64_t N,
                                         int interpolation, double oversampling, double cutoff,
                                         float* grad_rec, float* grad_rot, float* grad_shifts,
                                         const int32_t* pose_order, void* stream) {
    return project_back_saved<3>(grad_proj, out, derivatives, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, grad_rec, grad_rot, grad_shifts, pose_order, stream);
}

int b200proj_backproject_2d_forw(const float* proj, const float* weights, int64_t B, int64_t R,
                                 const float* rot, int64_t B_rot, const float* shifts,
                                 int64_t B_shift, int64_t P, int64_t N, int interpolation,
                                 double oversampling, double cutoff, float* data_rec,
                                 float* weight_rec, int accumulate, void* workspace, size_t workspace_bytes, void* stream) {
    return backproject_forw<2>(proj, weights, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, data_rec, weight_rec, accumulate, workspace, workspace_bytes, stream);
}
int b200proj_backproject_2d_to_3d_forw(const float* proj, const float* weights, int64_t B,
                                       int64_t R, const float* rot, int64_t B_rot,
                                       const float* shifts, int64_t B_shift, int64_t P, int64_t N,
                                       int interpolation, double oversampling, double cutoff,
                                       float* data_rec, float* weight_rec, int accumulate,                                        void* workspace, size_t workspace_bytes, void* stream) {
    return backproject_forw<3>(proj, weights, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, data_rec, weight_rec, accumulate, workspace, workspace_bytes, stream);
}

int b200proj_backproject_2d_back(const float* grad_data_rec, const float* grad_weight_rec,
                                 const float* proj, int64_t B, int64_t R, const float* rot,
                                 int64_t B_rot, const float* shifts, int64_t B_shift, int64_t P,
                                 int64_t N, int interpolation, double oversampling, double cutoff,
                                 float* grad_proj, float* grad_weights, float* grad_rot,
                                 float* grad_shifts, void* stream) {
    return backproject_back<2>(grad_data_rec, grad_weight_rec, proj, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, grad_proj, grad_weights, grad_rot, grad_shifts, nullptr, stream);
}
int b200proj_backproject_2d_to_3d_back(const float* grad_data_rec, const float* grad_weight_rec,
                                       const float* proj, int64_t B, int64_t R, const float* rot,
                                       int64_t B_rot, const float* shifts, int64_t B_shift,
                                       int64_t P, int64_t N, int interpolation,
                                       double oversampling, double cutoff, float* grad_proj,
                                       float* grad_weights, float* grad_rot, float* grad_shifts,
                                       const int32_t* pose_order, void* stream) {
    return backproject_back<3>(grad_data_rec, grad_weight_rec, proj, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, grad_proj, grad_weights, grad_rot, grad_shifts, pose_order, stream);
}

// ---- complex128 / float64 variants (same kernels instantiated for double) ----------------
int b200proj_project_2d_forw_f64(const double* rec, int64_t B, int64_t R, const double* rot, int64_t B_rot,
                             const double* shifts, int64_t B_shift, int64_t P, int64_t N,
                             int interpolation, double oversampling, double cutoff, double* out,
                             void* stream) {
    return project_forw<2>(rec, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, out, nullptr, stream);
}
int b200proj_project_3d_to_2d_forw_f64(const double* rec, int64_t B, int64_t R, const double* rot,
                                   int64_t B_rot, const double* shifts, int64_t B_shift, int64_t P,
                                   int64_t N, int interpolation, double oversampling, double cutoff,
                                   double* out, const int32_t* pose_order, void* stream) {
    return project_forw<3>(rec, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, out, pose_order, stream);
}

int b200proj_project_2d_back_f64(const double* grad_proj, const double* rec, int64_t B, int64_t R,
                             const double* rot, int64_t B_rot, const double* shifts, int64_t B_shift,
                             int64_t P, int64_t N, int interpolation, double oversampling,
                             double cutoff, double* grad_rec, double* grad_rot, double* grad_shifts,
                             void* stream) {
    return project_back<2>(grad_proj, rec, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, grad_rec, grad_rot, grad_shifts, nullptr, stream);
}
int b200proj_project_3d_to_2d_back_f64(const double* grad_proj, const double* rec, int64_t B, int64_t R,
                                   const double* rot, int64_t B_rot, const double* shifts,
                                   int64_t B_shift, int64_t P, int64_t N, int interpolation,
                                   double oversampling, double cutoff, double* grad_rec,
                                   double* grad_rot, double* grad_shifts, const int32_t* pose_order,
                                   void* stream) {
    return project_back<3>(grad_proj, rec, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, grad_rec, grad_rot, grad_shifts, pose_order, stream);
}

int b200proj_backproject_2d_forw_f64(const double* proj, const double* weights, int64_t B, int64_t R,
                                 const double* rot, int64_t B_rot, const double* shifts,
                                 int64_t B_shift, int64_t P, int64_t N, int interpolation,
                                 double oversampling, double cutoff, double* data_rec,
                                 double* weight_rec, int accumulate, void* workspace, size_t workspace_bytes, void* stream) {
    return backproject_forw<2>(proj, weights, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, data_rec, weight_rec, accumulate, workspace, workspace_bytes, stream);
}
int b200proj_backproject_2d_to_3d_forw_f64(const double* proj, const double* weights, int64_t B,
                                       int64_t R, const double* rot, int64_t B_rot,
                                       const double* shifts, int64_t B_shift, int64_t P, int64_t N,
                                       int interpolation, double oversampling, double cutoff,
                                       double* data_rec, double* weight_rec, int accumulate,                                        void* workspace, size_t workspace_bytes, void* stream) {
    return backproject_forw<3>(proj, weights, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, data_rec, weight_rec, accumulate, workspace, workspace_bytes, stream);
}

int b200proj_backproject_2d_back_f64(const double* grad_data_rec, const double* grad_weight_rec,
                                 const double* proj, int64_t B, int64_t R, const double* rot,
                                 int64_t B_rot, const double* shifts, int64_t B_shift, int64_t P,
                                 int64_t N, int interpolation, double oversampling, double cutoff,
                                 double* grad_proj, double* grad_weights, double* grad_rot,
                                 double* grad_shifts, void* stream) {
    return backproject_back<2>(grad_data_rec, grad_weight_rec, proj, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, grad_proj, grad_weights, grad_rot, grad_shifts, nullptr, stream);
}
int b200proj_backproject_2d_to_3d_back_f64(const double* grad_data_rec, const double* grad_weight_rec,
                                       const double* proj, int64_t B, int64_t R, const double* rot,
                                       int64_t B_rot, const double* shifts, int64_t B_shift,
                                       int64_t P, int64_t N, int interpolation,
                                       double oversampling, double cutoff, double* grad_proj,
                                       double* grad_weights, double* grad_rot, double* grad_shifts,
                                       const int32_t* pose_order, void* stream) {
    return backproject_back<3>(grad_data_rec, grad_weight_rec, proj, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, grad_proj, grad_weights, grad_rot, grad_shifts, pose_order, stream);
}

int b200proj_backproject_2d_to_3d_accumulate(const float* proj, const float* weights, int64_t B,
                                             int64_t R, const float* rot, int64_t B_rot,
                                             const float* shifts, int64_t B_shift, int64_t P,
                                             int64_t N, int interpolation, double oversampling,
                                             double cutoff, void* accumulator, void* stream) {
    return backproject_accumulate(proj, weights, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, accumulator, 0, -1, stream);
}

int b200proj_backproject_2d_to_3d_accumulate_ws(const float* proj, const float* weights, int64_t B,
                                                int64_t R, const float* rot, int64_t B_rot,
                                                const float* shifts, int64_t B_shift, int64_t P,
                                                int64_t N, int interpolation, double oversampling,
                                                double cutoff, void* accumulator, void* workspace, size_t workspace_bytes, void* stream) {
    return backproject_accumulate(proj, weights, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, accumulator, 0, -1, stream, workspace, workspace_bytes);
}

int b200proj_backproject_2d_to_3d_accumulate_slabs(const float* proj, const float* weights, int64_t B,
                                                   int64_t R, const float* rot, int64_t B_rot,
                                                   const float* shifts, int64_t B_shift, int64_t P,
                                                   int64_t N, int interpolation, double oversampling,
                                                   double cutoff, void* accumulator, int slab_first,
                                                   int slab_count, void* stream) {
    if (slab_count < 0) return fail(B200PROJ_ERR_ARGUMENT, "slab_count must be >= 1");
    return backproject_accumulate(proj, weights, B, R, rot, B_rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff, accumulator, slab_first, slab_count, stream);
}

int b200proj_accumulator_slab_plan(int64_t R, int32_t* slabs, int32_t* planes_per_slab) {
    g_error[0] = 0;
    if (R < 2 || (R % 2) != 0 || slabs == nullptr || planes_per_slab == nullptr)
        return fail(B200PROJ_ERR_ARGUMENT, "need an even boxsize >= 2 and two output pointers");
    const SlabPlan plan = slab_plan(R, true, true);
    *slabs = plan.slabs;
    *planes_per_slab = plan.planes;
    return B200PROJ_OK;
}

int b200proj_accumulator_slab_voxels(int64_t R, int slab_first, int slab_count, int64_t first_voxel[2], int64_t voxel_count[2]) {
    g_error[0] = 0;
    if (R < 2 || (R % 2) != 0 || first_voxel == nullptr || voxel_count == nullptr)
        return fail(B200PROJ_ERR_ARGUMENT, "need an even boxsize >= 2 and two output arrays");
    const SlabPlan plan = slab_plan(R, true, true);
    if (slab_first < 0 || slab_count < 1 || slab_first + slab_count > plan.slabs)
        return fail(B200PROJ_ERR_ARGUMENT, "slabs [%d, %d) outside the plan of %d slabs", slab_first, slab_first + slab_count, plan.slabs);
    // signed plane coordinates [z_a, z_b) of the slabs; plane z is stored at index z < 0 ? z + R : z
    const int64_t half = R / 2, plane = R * (R / 2 + 1);
    const int64_t z_a = -half + 1 + (int64_t)slab_first * plan.planes;
    int64_t z_b = z_a + (int64_t)slab_count * plan.planes;
    if (z_b > half + 1) z_b = half + 1;
    const int64_t neg_b = z_b < 0 ? z_b : 0, pos_a = z_a > 0 ? z_a : 0;
    first_voxel[0] = (z_a < neg_b) ? (z_a + R) * plane : 0;            // planes with negative coordinates
    voxel_count[0] = (z_a < neg_b) ? (neg_b - z_a) * plane : 0;
    first_voxel[1] = (pos_a < z_b) ? pos_a * plane : 0;                // planes with coordinates >= 0
    voxel_count[1] = (pos_a < z_b) ? (z_b - pos_a) * plane : 0;
    return B200PROJ_OK;
}

size_t b200proj_accumulator_bytes(int64_t B, int64_t R) {
    if (B < 1 || R < 2) return 0;
    return (size_t)B * (size_t)R * (size_t)R * (size_t)(R / 2 + 1) * sizeof(float4);
}

int b200proj_accumulator_fold_range(const void* accumulator, int64_t first_voxel, int64_t voxel_count,
                                    float* data_rec, float* weight_rec, int accumulate, void* stream) {
    g_error[0] = 0;
    if (accumulator == nullptr || data_rec == nullptr || weight_rec == nullptr)
        return fail(B200PROJ_ERR_ARGUMENT, "accumulator, data_reconstruction and weight_reconstruction are all required");
    if (first_voxel < 0 || voxel_count < 0) return fail(B200PROJ_ERR_ARGUMENT, "voxel range must be non-negative (first=%lld, count=%lld)", (long long)first_voxel, (long long)voxel_count);
    if (voxel_count == 0) return B200PROJ_OK;
    const size_t n = (size_t)voxel_count;
    const size_t blocks = (n + 255) / 256;
    fold_interleaved_kernel<<<(unsigned)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, (cudaStream_t)stream>>>(
        (const float4*)accumulator + first_voxel, (float2*)data_rec + first_voxel, weight_rec + first_voxel, n, accumulate != 0);
    return check_launch("fold_interleaved launch");
}

int b200proj_accumulator_fold_normalized(const void* accumulator, int64_t first_voxel, int64_t voxel_count,
                                         double eps, float* normalized, void* stream) {
    g_error[0] = 0;
    if (accumulator == nullptr || normalized == nullptr) return fail(B200PROJ_ERR_ARGUMENT, "accumulator and output are required");
    if (first_voxel < 0 || voxel_count < 0) return fail(B200PROJ_ERR_ARGUMENT, "voxel range must be non-negative (first=%lld, count=%lld)", (long long)first_voxel, (long long)voxel_count);
    if (!(eps > 0.0)) return fail(B200PROJ_ERR_ARGUMENT, "eps must be positive");
    if (voxel_count == 0) return B200PROJ_OK;
    const size_t n = (size_t)voxel_count;
    const size_t blocks = (n + 255) / 256;
    fold_normalized_kernel<<<(unsigned)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, (cudaStream_t)stream>>>(
        (const float4*)accumulator + first_voxel, (float2*)normalized + first_voxel, n, (float)eps);
    return check_launch("fold_normalized launch");
}

int64_t b200proj_cutoff_pack_index(int64_t N, double cutoff, int32_t* index) {
    g_error[0] = 0;
    if (N < 2 || (N % 2) != 0 || N > 2048 || std::isnan(cutoff)) { fail(B200PROJ_ERR_ARGUMENT, "need an even projection boxsize in [2, 2048] and a cutoff"); return -1; }
    // the kernels' own test (pixel_setup): kr*kr + kc*kc > float(cutoff)^2 in fp32 excludes a pixel
    const float rc = (float)cutoff, cutoff_sq = rc * rc;
    const int64_t Nh = N / 2 + 1;
    int64_t count = 0;
    for (int64_t i = 0; i < N; ++i) {
        const float kr = (float)((i <= N / 2) ? i : i - N);
        for (int64_t j = 0; j < Nh; ++j) {
            const float kc = (float)j;
            const bool inside = !(kr * kr + kc * kc > cutoff_sq);
            if (index != nullptr) index[i * Nh + j] = inside ? (int32_t)count : -1;
            count += inside ? 1 : 0;
        }
    }
    return count;
}

int b200proj_project_3d_to_2d_forw_packed(const float* rec, int64_t B, int64_t R, const float* rot,
                                          int64_t B_rot, const float* shifts, int64_t B_shift, int64_t P,
                                          int64_t N, int interpolation, double oversampling, double cutoff,
                                          float* out_packed, const int32_t* pack_index, int64_t pack_count,
                                          const int32_t* pose_order, void* stream) {
    Launch L;
    if (int rc = prepare(L, 3, B, R, B_rot, rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff)) return rc;
    if (rec == nullptr || out_packed == nullptr || pack_index == nullptr)
        return fail(B200PROJ_ERR_ARGUMENT, "reconstruction / output / pack_index pointer is NULL");
    if (pack_count != b200proj_cutoff_pack_index(N, cutoff, nullptr))
        return fail(B200PROJ_ERR_ARGUMENT, "pack_count %lld is not the number of pixels inside the cutoff (%lld)",
                    (long long)pack_count, (long long)b200proj_cutoff_pack_index(N, cutoff, nullptr));
    L.g.order = pose_order;
    L.g.pack_index = pack_index;
    L.g.pack_count = (int)pack_count;
    if (P == 0 || pack_count == 0) return B200PROJ_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (interpolation == B200PROJ_CUBIC)
        project_forw_kernel<3, true, float, true><<<L.grid, kBlockThreads, 0, s>>>((const float2*)rec, rot, shifts, (float2*)out_packed, L.g);
    else
        project_forw_kernel<3, false, float, true><<<L.grid, kBlockThreads, 0, s>>>((const float2*)rec, rot, shifts, (float2*)out_packed, L.g);
    return check_launch("project_forw (packed) launch");
}

int b200proj_reduction_rate_probe(int pattern, float* buffer, size_t buffer_bytes, int blocks, int iterations, void* stream) {
    g_error[0] = 0;
    if (buffer == nullptr || (reinterpret_cast<uintptr_t>(buffer) & 15u) != 0) return fail(B200PROJ_ERR_ARGUMENT, "buffer must be a 16-byte aligned device pointer");
    if (pattern < 0 || pattern > 5 || blocks < 1 || iterations < 1) return fail(B200PROJ_ERR_ARGUMENT, "pattern must be 0..5, blocks and iterations >= 1");
    const size_t unit = pattern <= 2 ? 16 : 8;
    const size_t units = buffer_bytes / unit;
    if (units < 16 || units > 0xffffffffull) return fail(B200PROJ_ERR_LIMIT, "buffer of %zu bytes holds too few or too many units", buffer_bytes);
    cudaStream_t s = (cudaStream_t)stream;
    switch (pattern) {
        case 0: reduction_rate_kernel<0><<<blocks, 256, 0, s>>>(buffer, (unsigned)units, iterations); break;
        case 1: reduction_rate_kernel<1><<<blocks, 256, 0, s>>>(buffer, (unsigned)units, iterations); break;
        case 2: reduction_rate_kernel<2><<<blocks, 256, 0, s>>>(buffer, (unsigned)units, iterations); break;
        case 3: reduction_rate_kernel<3><<<blocks, 256, 0, s>>>(buffer, (unsigned)units, iterations); break;
        case 4: reduction_rate_kernel<4><<<blocks, 256, 0, s>>>(buffer, (unsigned)units, iterations); break;
        default: reduction_rate_kernel<5><<<blocks, 256, 0, s>>>(buffer, (unsigned)units, iterations); break;
    }
    return check_launch("reduction_rate_probe launch");
}

int b200proj_reduction_rate_probe_streaming(float* target, size_t target_bytes, size_t window_bytes,
                                            const float* source, size_t source_bytes, int blocks,
                                            int iterations, int evict_last, void* stream) {
    g_error[0] = 0;
    if (target == nullptr || (reinterpret_cast<uintptr_t>(target) & 15u) != 0 || source == nullptr || (reinterpret_cast<uintptr_t>(source) & 7u) != 0)
        return fail(B200PROJ_ERR_ARGUMENT, "target must be a 16-byte and source an 8-byte aligned device pointer");
    if (blocks < 1 || iterations < 1) return fail(B200PROJ_ERR_ARGUMENT, "blocks and iterations must be >= 1");
    const size_t units = target_bytes / 16, window = window_bytes / 16, src_units = source_bytes / 8;
    if (window < 16 || units < window || units > 0xffffffffull || src_units < 256 || src_units > 0xffffffffull)
        return fail(B200PROJ_ERR_LIMIT, "target of %zu bytes, window of %zu bytes or source of %zu bytes out of range", target_bytes, window_bytes, source_bytes);
    if (evict_last)
        reduction_stream_kernel<true><<<blocks, 256, 0, (cudaStream_t)stream>>>(target, (unsigned)units, (unsigned)window,
                                                                               reinterpret_cast<const float2*>(source), (unsigned)src_units, iterations);
    else
        reduction_stream_kernel<false><<<blocks, 256, 0, (cudaStream_t)stream>>>(target, (unsigned)units, (unsigned)window,
                                                                                reinterpret_cast<const float2*>(source), (unsigned)src_units, iterations);
    return check_launch("reduction_rate_probe_streaming launch");
}

int b200proj_accumulator_fold(const void* accumulator, int64_t B, int64_t R, float* data_rec,
                              float* weight_rec, int accumulate, void* stream) {
    if (B < 1 || R < 2 || (R % 2) != 0) return fail(B200PROJ_ERR_ARGUMENT, "batch size must be >= 1 and the boxsize even (B=%lld, R=%lld)", (long long)B, (long long)R);
    return b200proj_accumulator_fold_range(accumulator, 0, B * R * R * (R / 2 + 1), data_rec, weight_rec, accumulate, stream);
}

int b200proj_pad_fftshift(const float* real, int64_t batch, int dims, int64_t n, int64_t m, float* out, void* stream) {
    return pad_shift(real, batch, dims, n, m, 1, out, stream);
}
int b200proj_pad_fftshift_f64(const double* real, int64_t batch, int dims, int64_t n, int64_t m, double* out, void* stream) {
    return pad_shift(real, batch, dims, n, m, 1, out, stream);
}
int b200proj_ifftshift_crop(const float* full, int64_t batch, int dims, int64_t m, int64_t n, float* out, void* stream) {
    return pad_shift(full, batch, dims, n, m, 0, out, stream);
}
int b200proj_ifftshift_crop_f64(const double* full, int64_t batch, int dims, int64_t m, int64_t n, double* out, void* stream) {
    return pad_shift(full, batch, dims, n, m, 0, out, stream);
}

int b200proj_pose_order_3d(const float* rot, int64_t B, int64_t B_rot, int64_t P, int32_t* order, void* stream) {
    return pose_order_3d(rot, B, B_rot, P, order, stream);
}
int b200proj_pose_order_3d_f64(const double* rot, int64_t B, int64_t B_rot, int64_t P, int32_t* order, void* stream) {
    return pose_order_3d(rot, B, B_rot, P, order, stream);
}

int b200proj_backproject_2d_to_3d_forw_noalloc(const float* proj, const float* weights, int64_t B,
                                               int64_t R, const float* rot, int64_t B_rot,
                                               const float* shifts, int64_t B_shift, int64_t P,
                                               int64_t N, int interpolation, double oversampling,
                                               double cutoff, float* data_rec, float* weight_rec,
                                               int accumulate, void* stream) {
    Launch L;
    if (int rc = prepare(L, 3, B, R, B_rot, rot, shifts, B_shift, P, N, interpolation, oversampling, cutoff)) return rc;
    if (proj == nullptr || weights == nullptr || data_rec == nullptr || weight_rec == nullptr)
        return fail(B200PROJ_ERR_ARGUMENT, "projections, weights, data_reconstruction and weight_reconstruction are all required");
    if (R != b200proj_rec_boxsize(N, oversampling))
        return fail(B200PROJ_ERR_ARGUMENT, "reconstruction boxsize %lld does not match ceil(N*oversampling) rounded up to even = %lld",
                    (long long)R, (long long)b200proj_rec_boxsize(N, oversampling));
    if ((long long)L.rec_count > kNoAllocMaxVoxels)
        return fail(B200PROJ_ERR_LIMIT, "B*R*R*(R/2+1) = %lld voxels exceed the built-in scratch of %lld voxels (box 64, one batch item); "
                    "use b200proj_backproject_2d_to_3d_forw with a caller-provided workspace",
                    (long long)L.rec_count, kNoAllocMaxVoxels);
    float4* acc = nullptr;
    if (int rc = noalloc_scratch(&acc)) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    // the scratch keeps the previous call's sums: clear the part this call uses
    if (int rc = zero_async(acc, L.rec_count * sizeof(float4), s)) return rc;
    if (P > 0) {
        if (interpolation == B200PROJ_CUBIC)
            backproject_forw_interleaved_kernel<3, true><<<L.grid, kBlockThreads, 0, s>>>((const float2*)proj, weights, rot, shifts, acc, L.g);
        else
            backproject_forw_interleaved_kernel<3, false><<<L.grid, kBlockThreads, 0, s>>>((const float2*)proj, weights, rot, shifts, acc, L.g);
        if (int rc = check_launch("backproject_forw (built-in scratch) launch")) return rc;
    }
    const size_t blocks = (L.rec_count + 255) / 256;
    fold_interleaved_kernel<<<(unsigned)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, s>>>(acc, (float2*)data_rec, weight_rec, L.rec_count, accumulate != 0);
    return check_launch("fold_interleaved launch");
}

}  // extern "C"
