// Brick-stationary kernels (fp32; 3D, and 2D with cubic taps): the volume is cut into bricks that fit shared
// memory, a block keeps one brick and walks over the slices, handling the pixels whose sample position
// lies in its brick.  The plain kernels (fourier_slice_kernels.cuh) keep the pixels and fetch the taps
// of every pixel through L1: 16 rows of a cubic footprint are 13 cache lines per pixel, and the L1TEX
// data pipe retires about one a clock.  Here a brick is staged once per work item and the taps of all
// its pixels, of all slices, come from shared memory without bank conflicts, 16 lanes = 128 bytes a
// wavefront: 4 wavefronts per cubic pixel instead of 13-18.  Measured on B200: 10,000 slices of 128 x 65
// from a box-256 volume, cubic, 3.95 -> 1.77 ms (62 -> 27 ps per pixel; data pipe 75 %, issue 69 %), with
// records 8.9 -> 4.0 ms for 4,096 slices of 256 x 129 from a box-512 volume; linear 1.09 -> 0.97 ms.
//
// Bricks of 17 x 17 x 16 sample positions (cubic): with the halo 20 x 20 x 19 voxels = 61 KB, three
// blocks (24 warps, 80 registers) per SM.  Smaller bricks meet a slice in too few pixels (here 40) to
// pay for finding them.
//
// A call runs as two launches:
//   brick_setup_kernel   per slice a 64-byte record (plane, half-plane, matrix, its rows); per brick its work items
//   brick_*_kernel       persistent blocks take items (brick, range of slices) from a ticket counter
// Nothing waits on another block.
#pragma once

#include "fourier_slice_kernels.cuh"

namespace b200proj {

// Sample positions of a brick (units of voxels); Z = 0: a tile of a 2D reconstruction.
template <int X, int Y, int Z>
struct BrickDims {
    static constexpr int x = X, y = Y, z = Z, kDim = Z > 0 ? 3 : 2;
};
// 2D tiles of 61 x 61 (64 x 64 with the halo, 32 KB): all slices of a half-plane meet a tile, in rows of some 30 pixels,
// so that the walk costs less than in 3D (500 slices of 128 x 65 from each of eight references, cubic: 0.755 -> 0.350 ms).
// Linear taps have a halo of one voxel, and 64 registers are enough: bricks of 15 x 15 x 16 (16 x 16 x 17 voxels, 35 KB) make room for four
// blocks per SM.  Linear, 3,001 slices of 180 x 91 478 -> 443 us, 8,000 of 128 x 65 from a box-256 volume 816 -> 777, records of 2,000 of
// 200 x 101 548 -> 521; 15 x 15 x 20 444, 747, 547; 19 x 19 x 18 and three blocks 473, 770, 563; 23 x 23 x 21 and two 561; 15 x 15 x 13 and five 463.
template <int DIM, bool CUBIC>
struct GatherBrickOf { using type = BrickDims<17, 17, 16>; };
template <>
struct GatherBrickOf<3, false> { using type = BrickDims<15, 15, 16>; };
template <bool CUBIC>
struct GatherBrickOf<2, CUBIC> { using type = BrickDims<61, 61, 0>; };
template <int DIM, bool CUBIC>
using GatherBrick = typename GatherBrickOf<DIM, CUBIC>::type;
constexpr int kBrickSlots = 8;                              // slices a warp takes at a time
constexpr float kBrickSlack = 0.06f;                        // slack of the linear estimates, in voxels

// The samples of a rotated slice lie inside a ball, those of a matrix that stretches by s inside one s times as large.  The
// bricks are listed in shells: 0 for rotations, l for slices that stretch by up to kStretch[l]; the shells beyond 0 are
// worked on only when a call has slices that need them.  (Rotations alone and all else pixel by pixel, one slice per
// block: 10,000 cubic slices of 128 x 65, all stretched by 1.01, took 6.84 ms where the plain kernel takes 3.96, from a
// box-512 volume 14.2 against 3.34.)
constexpr int kShells = 5;
__host__ __device__ constexpr float brick_stretch(int shell) { return shell == 0 ? 1.f : shell == 1 ? 1.1f : shell == 2 ? 1.3f : shell == 3 ? 1.6f : 2.f; }

// What the host derives from the sizes (see brick_plan in b200proj.cu).
struct BrickPlan {
    int n[3];               // bricks along x (column), y (row), z (plane)
    int d[3];               // sample positions of a brick along them
    int lo[3];              // first sample position of the grid
    float reach;            // distance from the origin of the farthest sample of a rotated slice
    int shells;             // of the grid
    int at[kShells];        // where their work items start in the list
    int keep;               // bricks beyond this coordinate are left out (scatters: nothing of them is stored)
    float density;          // expected pixels per brick and slice: density / max(r, ...) at radius r (2D: density)
    float per_slice;        // pixels of a slice inside the cutoff
    float target;           // pixels a work item should hold
    int max_extra;          // items beyond one per brick that fit the list of a shell
    int wait_ms;            // after which a scatter's wait gives up
};

// Workspace layout: int header[20] {-, -, ticket, gathers: pixels outside the cutoff, scatters: 1 when a wait gave up; last
// shell in use, -, -, -; items of each shell; extra items of each shell}, int4 items[shells], float4 records[4 * B * P],
// float2 shifts[B * P], int outside[N * Nh].
struct BrickWork {
    int* header;
    int4* items;
    float4* recs;
    float2* shifts;
    int* outside;
};

// A slice's record.  The columns a and b of its matrix map a pixel to a sample: x = os (kc a + kr b).
struct SliceRec {           // 64 bytes
    float4 a;               // unit normal of the plane (NaN: the slice is not for the bricks), then the unit vector
    float4 b;               // in the plane along which kc grows at fixed kr b (2 more), a.x, a.y
    float4 c;               // a.z, b.x, b.y, b.z
    float4 d;               // v with v.a = 0, v.b = 1: a sample x of the slice is of row v.x / os; -
};

// Plane, half-plane and shell of a slice; -1: not for the bricks.  Any two columns that are far from parallel and stretch by
// no more than the last shell will do (then the linear estimates of the walk hold with their slack: they lose at most
// a factor of 25 to cancellation, of 1e-7 of some 2,000 voxels).
template <int DIM>
__device__ __forceinline__ int brick_slice_fit(const BrickPlan& pl, const float (&a)[3], const float (&b)[3], float (&n)[3], float (&h)[3], float (&v)[3]) {
    const float aa = a[0] * a[0] + a[1] * a[1] + a[2] * a[2], bb = b[0] * b[0] + b[1] * b[1] + b[2] * b[2], ab = a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
    const float det = aa * bb - ab * ab, diff = aa - bb;
    const float most = 0.5f * (aa + bb + sqrtf(diff * diff + 4.f * ab * ab)), least = det / most;       // squared singular values
    if (!(most <= 4.f && least >= 0.04f * most && least >= 0.01f)) return -1;
    const float inv = rsqrtf(det), t = ab / bb, len = rsqrtf(det / bb);
    n[0] = (a[1] * b[2] - a[2] * b[1]) * inv;
    n[1] = (a[2] * b[0] - a[0] * b[2]) * inv;
    n[2] = DIM == 3 ? (a[0] * b[1] - a[1] * b[0]) * inv : 0.f;         // 2D: every tile is in the plane
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        h[q] = (a[q] - t * b[q]) * len;
        v[q] = (aa * b[q] - ab * a[q]) / det;
    }
    const float far = sqrtf(most) * pl.reach;
    for (int l = 0; l < pl.shells; ++l)
        if (far <= brick_stretch(l) * pl.reach + 0.9f) return l;
    return -1;
}
__device__ __forceinline__ bool brick_has_slice(const BrickWork& ws, int k) { return !isnan(__ldg(&ws.recs[4 * (size_t)k].x)); }

// Shell of a brick; -1: none.
__device__ __forceinline__ int brick_shell(const BrickPlan& pl, int bx, int by, int bz, float& r_center) {
    const int at[3] = {bx, by, bz};
    float near2 = 0.f, mid2 = 0.f;
    bool out = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int lo = pl.lo[a] + at[a] * pl.d[a];
        const float x = (float)lo, n = fmaxf(fmaxf(x, -(x + (float)pl.d[a])), 0.f), c = x + 0.5f * (float)pl.d[a];
        out = out || lo - 1 > pl.keep || lo + pl.d[a] + 1 < -pl.keep;
        near2 += n * n;
        mid2 += c * c;
    }
    r_center = sqrtf(mid2);
    if (out) return -1;
    for (int l = 0; l < pl.shells; ++l) {
        const float ball = brick_stretch(l) * pl.reach + 1.f;
        if (near2 <= ball * ball) return l;
    }
    return -1;
}

// The work items of a call: those of the shells in use.
__device__ __forceinline__ int brick_items(const BrickWork& ws) {
    const int last = __ldg(ws.header + 4);
    int n = 0;
#pragma unroll
    for (int l = 0; l < kShells; ++l) {
        const int here = __ldg(ws.header + 8 + l);
        n += l <= last ? here : 0;
    }
    return n;
}
__device__ __forceinline__ int4 brick_item(const BrickWork& ws, const BrickPlan& pl, int item) {
    int at = -1;
#pragma unroll
    for (int l = 0; l < kShells; ++l) {
        const int n = __ldg(ws.header + 8 + l);
        if (at < 0 && item < n) at = pl.at[l] + item;
        item -= n;
    }
    return __ldg(ws.items + at);
}

// The pixels outside the cutoff, by one block of 256 threads: their offsets in a slice, row by row.
__device__ __forceinline__ void brick_list_outside(const SliceGeom& g, BrickWork ws) {
    __shared__ int row_at[2049];
    // first column outside: rad is monotonic in j, the estimate is at most one column late
    auto first_out = [&](int i) {
        const float kr = (float)((i <= g.N / 2) ? i : i - g.N), kr2 = mul_rn(kr, kr), room = g.cutoff_sq - kr2;
        int j = room > 0.f ? max(0, (int)fminf(sqrtf(room), (float)g.Nh) - 1) : 0;
        while (j < g.Nh && !(add_rn(kr2, mul_rn((float)j, (float)j)) > g.cutoff_sq)) ++j;
        return j;
    };
    // row_at[i + 1] = pixels of rows 0 .. i: 256 threads with a run of rows each
    __shared__ int warp_rows[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, per = (g.N + 255) / 256, row0 = (int)threadIdx.x * per, row1 = min(row0 + per, g.N);
    int sum = 0;
    for (int i = row0; i < row1; ++i) sum += g.Nh - first_out(i);
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
    }
    if (lane == 31) warp_rows[warp] = incl;
    __syncthreads();
    int at = incl - sum;
    for (int w = 0; w < warp; ++w) at += warp_rows[w];
    if (threadIdx.x == 0) row_at[0] = 0;
    for (int i = row0; i < row1; ++i) row_at[i + 1] = at += g.Nh - first_out(i);
    __syncthreads();
    if (threadIdx.x == 0) ws.header[3] = row_at[g.N];
    for (int i = warp; i < g.N; i += 8) {
        const int first = row_at[i], n = row_at[i + 1] - first;
        for (int q = lane; q < n; q += 32) ws.outside[first + q] = i * g.Nh + g.Nh - n + q;
    }
}

// Slice records (a thread per slice) and work items (a thread per brick and batch item).  The header
// is zero on entry.  A brick's slices are split over as many items as bring one near pl.target pixels for
// uniformly distributed poses (the density of pixels falls as 1 / r); a shell's list has room for one item per
// brick plus max_extra, of which a brick takes what is left.
// Neighbouring bricks are neighbours in the list, so that they run at the same time: the runs of pixels that
// they write into a row of a slice then meet in L2 before the row's sectors leave it.
template <int DIM>
__global__ void __launch_bounds__(256)
brick_setup_kernel(const float* __restrict__ rot, const float* __restrict__ shifts, BrickWork ws, const SliceGeom g, const BrickPlan pl, int B, int list_outside, Gate gate) {
    if (gate.shut()) return;
    // block 0: the pixels outside the cutoff; then one block per cluster of bricks and batch item; then the slices
    if (blockIdx.x == 0) {
        if (list_outside) brick_list_outside(g, ws);
        return;
    }
    const int cx = (pl.n[0] + 7) / 8, cy = (pl.n[1] + 7) / 8, cz = (pl.n[2] + 3) / 4, clusters = cx * cy * cz * B;
    if ((int)blockIdx.x > clusters) {
        const int t = ((int)blockIdx.x - 1 - clusters) * 256 + (int)threadIdx.x;
        int shell = 0;
        if (t < g.BP) {
            const int b = t / g.P, p = t - b * g.P;
            const float* rm = pose_rot<DIM>(g, rot, b, p);
            const float ma[3] = {__ldg(rm + 0), __ldg(rm + DIM), DIM == 3 ? __ldg(rm + 6) : 0.f}, mb[3] = {__ldg(rm + 1), __ldg(rm + DIM + 1), DIM == 3 ? __ldg(rm + 7) : 0.f};
            float n[3] = {0.f, 0.f, 0.f}, h[3] = {0.f, 0.f, 0.f}, v[3] = {0.f, 0.f, 0.f};
            shell = brick_slice_fit<DIM>(pl, ma, mb, n, h, v);
            if (shell < 0) n[0] = __int_as_float(0x7fffffff);
            ws.recs[4 * (size_t)t + 0] = make_float4(n[0], n[1], n[2], h[0]);
            ws.recs[4 * (size_t)t + 1] = make_float4(h[1], h[2], ma[0], ma[1]);
            ws.recs[4 * (size_t)t + 2] = make_float4(ma[2], mb[0], mb[1], mb[2]);
            ws.recs[4 * (size_t)t + 3] = make_float4(v[0], v[1], v[2], 0.f);
            if (g.has_shift) {
                const float* s = pose_shift(g, shifts, b, p);
                ws.shifts[t] = make_float2(__ldg(s), __ldg(s + 1));
            }
        }
        shell = __reduce_max_sync(0xffffffffu, shell);
        if (shell > 0 && (threadIdx.x & 31) == 0) atomicMax(ws.header + 4, shell);
        return;
    }
    // work items: a block takes a cluster of 8 x 8 x 4 neighbouring bricks of one batch item
    __shared__ int warp_sum[8], shell_sum[kShells][8], block_at[kShells], upto[257], code[256], start[256];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int b = ((int)blockIdx.x - 1) / (cx * cy * cz), k = (int)blockIdx.x - 1 - b * (cx * cy * cz);
    const int bx = k % cx * 8 + (threadIdx.x & 7), by = k / cx % cy * 8 + (threadIdx.x >> 3 & 7), bz = k / (cx * cy) * 4 + (threadIdx.x >> 6);
    int parts = 0;
    float r;
    const int mine = bx < pl.n[0] && by < pl.n[1] && bz < pl.n[2] ? brick_shell(pl, bx, by, bz, r) : -1;
    if (mine >= 0) {
        const float expected = fminf(DIM == 3 ? pl.density / fmaxf(r, 0.42f * (float)pl.d[0]) : pl.density, pl.per_slice) * (float)g.P;
        parts = max(1, min((int)(expected / pl.target + 0.5f), (g.P + 31) / 32));
    }
    auto scan = [&](int n) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, n, o);
            if (lane >= o) n += up;
        }
        return n;
    };
    // what the list of extra items has room for, and the place of the brick's first item in its shell's list
    int place = 0;
    for (int l = 0; l < pl.shells; ++l) {
        int sum = 0;
        if (__any_sync(0xffffffffu, mine == l)) {
            const int extra = mine == l ? parts - 1 : 0, extra_upto = scan(extra);
            int taken = 0;
            if (lane == 31 && extra_upto > 0) taken = atomicAdd(ws.header + 8 + kShells + l, extra_upto);
            taken = __shfl_sync(0xffffffffu, taken, 31) + extra_upto - extra;
            if (mine == l) parts = 1 + max(0, min(extra, pl.max_extra - taken));
            const int n = mine == l ? parts : 0, upto_me = scan(n);
            if (mine == l) place = upto_me - n;
            sum = __shfl_sync(0xffffffffu, upto_me, 31);
        }
        if (lane == l) shell_sum[l][warp] = sum;
    }
    const int incl = scan(parts);
    if (lane == 31) warp_sum[warp] = incl;
    if (__syncthreads_or(parts) == 0) return;
    if (threadIdx.x < pl.shells) {
        int sum = 0;
        for (int w = 0; w < 8; ++w) { const int n = shell_sum[threadIdx.x][w]; shell_sum[threadIdx.x][w] = sum; sum += n; }
        if (sum > 0) block_at[threadIdx.x] = pl.at[threadIdx.x] + atomicAdd(ws.header + 8 + threadIdx.x, sum);
    } else if (threadIdx.x == 32) {
        int sum = 0;
        for (int w = 0; w < 8; ++w) { const int n = warp_sum[w]; warp_sum[w] = sum; sum += n; }
        upto[256] = sum;
    }
    __syncthreads();
    upto[threadIdx.x] = warp_sum[warp] + incl;
    code[threadIdx.x] = bx | by << 10 | bz << 20;
    start[threadIdx.x] = mine >= 0 ? block_at[mine] + shell_sum[mine][warp] + place : 0;
    __syncthreads();
    // a brick's slices in `parts` nearly equal shares; all threads write items, a thread finds the brick of its item by search
    for (int o = threadIdx.x; o < upto[256]; o += 256) {
        int t0 = 0;
#pragma unroll
        for (int step = 128; step > 0; step >>= 1)
            if (upto[t0 + step - 1] <= o) t0 += step;
        const int before = t0 ? upto[t0 - 1] : 0, n = upto[t0] - before, q = o - before;
        const int share = g.P / n, more = g.P - share * n, first = b * g.P + q * share + min(q, more);
        ws.items[start[t0] + q] = make_int4(code[t0], b, first, first + share + (q < more ? 1 : 0));
    }
}

// Shared-memory layout of a staged brick: 4 x 4 cells of (x, y) are contiguous, so that the place of a voxel
// modulo 16 is its class (x & 3) + 4 (y & 3).  A cubic footprint holds every class once per plane; lane l takes
// the columns and rows of its footprint in an order that starts at class (l & 3, (l >> 2) & 3), so that at
// every step the 16 lanes of a half-warp hold 16 different classes = 16 different 8-byte banks, wherever
// their pixels lie.
template <int DIM, bool CUBIC>
struct BrickShape {
    using D = GatherBrick<DIM, CUBIC>;
    static constexpr int T = CUBIC ? 4 : 2;
    static constexpr int TX = ((D::x + T - 1) + 3) / 4 * 4, TY = ((D::y + T - 1) + 3) / 4 * 4, TZ = DIM == 3 ? D::z + T - 1 : 1;
    static constexpr int kRowCells = TX / 4 * 16;            // voxels of four rows
    static constexpr int kPlane = TX * TY;
    static constexpr int kVoxels = kPlane * TZ;
};
__device__ __forceinline__ int brick_off_x(int x) { return x + 12 * (x >> 2); }
template <typename S>
__device__ __forceinline__ int brick_off_y(int y) { return 4 * (y & 3) + S::kRowCells * (y >> 2); }

// Stage the brick: voxel (x, y, z) of it is tap (X0 - o + x, Y0 - o + y, Z0 - o + z), o = 1 for cubic, read with
// the gather's rules (Friedel mirror with conjugation, clamping), so that edges need no further care.
template <int DIM, bool CUBIC>
__device__ __forceinline__ void brick_stage(const SliceGeom& g, const float2* __restrict__ vol, float2* sm, int X0, int Y0, int Z0) {
    using S = BrickShape<DIM, CUBIC>;
    constexpr int o = CUBIC ? 1 : 0, kRows = kBlockThreads / S::TX;      // rows staged at a time
    const int x = (int)threadIdx.x % S::TX, first = (int)threadIdx.x / S::TX;
    if (first >= kRows) return;
    bool m;
    const int col = gather_col<CUBIC>(g, X0 - o + x, m);
    const int ox = brick_off_x(x);
    int y = first, z = 0;
#pragma unroll 4
    for (int n = first; n < S::TY * S::TZ; n += kRows) {
        const int row = gather_line<CUBIC>(g, Y0 - o + y, m), pln = DIM == 3 ? gather_line<CUBIC>(g, Z0 - o + z, m) : 0;
        float2 v = __ldg(vol + ((pln * g.R + row) * g.Rh + col));
        if (m) v.y = -v.y;
        sm[z * S::kPlane + brick_off_y<S>(y) + ox] = v;
        y += kRows;
        if (y >= S::TY) { y -= S::TY; ++z; }
    }
}

template <typename F>
__device__ __forceinline__ void rotate4(F (&w)[4], int t0) {      // w[s] <- w[(s + t0) & 3]
    if (t0 & 1) { const F x = w[0]; w[0] = w[1]; w[1] = w[2]; w[2] = w[3]; w[3] = x; }
    if (t0 & 2) { F x = w[0]; w[0] = w[2]; w[2] = x; x = w[1]; w[1] = w[3]; w[3] = x; }
}

// Value (and derivatives) at (lx + fx, ly + fy, lz + fz) of the staged brick, all of it in this lane.
template <int DIM, bool CUBIC, bool WITH_DERIV>
__device__ __forceinline__ void brick_gather(const float2* sm, int lx, int ly, int lz, float fx, float fy, float fz,
                                             float2& val, float2& gc, float2& gr, float2& gd) {
    using S = BrickShape<DIM, CUBIC>;
    using u64 = unsigned long long;
    const int lane = threadIdx.x & 31;
    constexpr int T = S::T, TD = DIM == 3 ? T : 1;
    int ox[T], oy[T];                // byte offsets of the columns and rows, in this lane's order
    u64 wx[T], wy[T], wz[T], dx[T], dy[T], dz[T];
    const int base = (lz * S::kPlane + (ly >> 2) * S::kRowCells + (lx >> 2) * 16) * 8;
    if constexpr (CUBIC) {
        // the tap of class a lies in the first cell of the footprint when a >= (first tap's class), else in the next one
        float w[4];
        const int rx = lx & 3, ry = ly & 3, tx = (lane - lx) & 3, ty = ((lane >> 2) - ly) & 3;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int ax = (lane + s) & 3, ay = ((lane >> 2) + s) & 3;
            ox[s] = ax * 8 + (ax < rx ? 128 : 0) + base;
            oy[s] = ay * 32 + (ay < ry ? S::kRowCells * 8 : 0);
        }
        cubic_weights(fx, w);
        rotate4(w, tx);
#pragma unroll
        for (int s = 0; s < 4; ++s) wx[s] = pack2(w[s], w[s]);
        cubic_weights(fy, w);
        rotate4(w, ty);
#pragma unroll
        for (int s = 0; s < 4; ++s) wy[s] = pack2(w[s], w[s]);
        cubic_weights(fz, w);
#pragma unroll
        for (int s = 0; s < 4; ++s) wz[s] = pack2(w[s], w[s]);
        if (WITH_DERIV) {
            cubic_dweights(fx, w);
            rotate4(w, tx);
#pragma unroll
            for (int s = 0; s < 4; ++s) dx[s] = pack2(w[s], w[s]);
            cubic_dweights(fy, w);
            rotate4(w, ty);
#pragma unroll
            for (int s = 0; s < 4; ++s) dy[s] = pack2(w[s], w[s]);
            cubic_dweights(fz, w);
#pragma unroll
            for (int s = 0; s < 4; ++s) dz[s] = pack2(w[s], w[s]);
        }
    } else {
        ox[0] = base + (lx & 3) * 8;
        ox[1] = ox[0] + ((lx & 3) == 3 ? 128 - 24 : 8);
        oy[0] = (ly & 3) * 32;
        oy[1] = oy[0] + ((ly & 3) == 3 ? S::kRowCells * 8 - 96 : 32);
        wx[0] = pack2(1.f - fx, 1.f - fx); wx[1] = pack2(fx, fx);
        wy[0] = pack2(1.f - fy, 1.f - fy); wy[1] = pack2(fy, fy);
        wz[0] = pack2(1.f - fz, 1.f - fz); wz[1] = pack2(fz, fz);
        dx[0] = dy[0] = dz[0] = pack2(-1.f, -1.f);
        dx[1] = dy[1] = dz[1] = pack2(1.f, 1.f);
    }
    const char* smb = reinterpret_cast<const char*>(sm);
    u64 v2 = 0ull, c2 = 0ull, r2 = 0ull, d2 = 0ull;
#pragma unroll
    for (int a = 0; a < T; ++a) {
        u64 A = 0ull, Bq = 0ull, Dq = 0ull;
#pragma unroll
        for (int b = 0; b < T; ++b) {
            const char* col = smb + (ox[a] + oy[b]);
            u64 s = 0ull, sd = 0ull;
#pragma unroll
            for (int k = 0; k < TD; ++k) {
                const u64 v = *reinterpret_cast<const u64*>(col + k * S::kPlane * 8);
                s = DIM == 3 ? fma2(wz[k], v, s) : v;
                if (WITH_DERIV && DIM == 3) sd = fma2(dz[k], v, sd);
            }
            A = fma2(wy[b], s, A);
            if (WITH_DERIV) {
                Bq = fma2(dy[b], s, Bq);
                if (DIM == 3) Dq = fma2(wy[b], sd, Dq);
            }
        }
        v2 = fma2(wx[a], A, v2);
        if (WITH_DERIV) {
            c2 = fma2(dx[a], A, c2);
            r2 = fma2(wx[a], Bq, r2);
            if (DIM == 3) d2 = fma2(wx[a], Dq, d2);
        }
    }
    unpack2(v2, val.x, val.y);
    if (WITH_DERIV) {
        unpack2(c2, gc.x, gc.y);
        unpack2(r2, gr.x, gr.y);
        unpack2(d2, gd.x, gd.y);
    }
}

// A warp's working set of the slice walk.
struct BrickWarp {
    uint2 segs[64];                 // rows of slices: {slot << 16 | (kr & 0xffff), ja << 16 | length}
    float4 slots[kBrickSlots][2];   // the slices' matrices and shifts {a.x, a.y, a.z, b.x}, {b.y, b.z, shift}
    int slice[kBrickSlots];         // and their indices
};

template <int WARPS, int HITS>
struct BrickBlock {
    static constexpr int kWalkers = WARPS, kHits = HITS;
    int nhits, next, item;
    int hits[HITS];                 // slices whose half-plane meets the brick
    BrickWarp warp[WARPS];
};

// The slice walk of one work item: calls body(active, slice record slot, i, j, pixel, lx, ly, lz) with all 32
// lanes for windows of 32 candidate pixels; `active` lanes hold a pixel whose sample position lies in the brick.
// Every pixel of the item's slices inside the brick is visited exactly once.
//   1. all threads test the slices' planes and half-planes (columns j >= 0) against the brick,
//   2. a warp takes a few slices from the list of hits and flattens their rows, one row per lane: row kr meets the
//      brick in one run of columns, clipped with linear estimates plus slack,
//   3. the non-empty runs of 32 rows are flattened into one index space, so that the windows are full although
//      a slice has only some 40 pixels in a brick and a row 5; each candidate is then tested exactly.
// The whole block walks together, or (BLOCK::kWalkers == 1) every warp by itself over each `parts`-th slice,
// so that it never waits for another warp.
template <typename D, typename BLOCK, typename Body>
__device__ __forceinline__ void brick_walk(const SliceGeom& g, const float4* __restrict__ recs, const float2* __restrict__ shifts, BLOCK& sb,
                                           int X0, int Y0, int Z0, int first, int last, int part, int parts, Body body) {
    constexpr bool kAlone = BLOCK::kWalkers == 1;
    constexpr int kThreads = BLOCK::kWalkers * 32;
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = kAlone ? 0 : threadIdx.x >> 5, thread = kAlone ? lane : threadIdx.x;
    const unsigned upto = 0xffffffffu >> (31 - lane);               // lanes up to this one
    BrickWarp& sw = sb.warp[warp];
    const float hx = 0.5f * D::x, hy = 0.5f * D::y, hz = 0.5f * D::z;
    const float cx = (float)X0 + hx, cy = (float)Y0 + hy, cz = (float)Z0 + hz;
    const float osf = (float)g.os, inv_os = 1.f / osf;
    const int grab = D::kDim == 3 ? max(1, min(kBrickSlots, (int)(2.f * osf))) : 1;       // slices with about 32 rows in the brick
    for (int k_next = first + part; k_next < last;) {
        if (!kAlone) {
            __syncthreads();
            if (thread == 0) { sb.nhits = 0; sb.next = 0; }
            __syncthreads();
        }
        int nhits = 0;
        do {            // as many slices as the list of hits has room for, whatever the tests say
            for (int room = (BLOCK::kHits - nhits) / kThreads; room > 0 && k_next < last; --room, k_next += kThreads * parts) {
                const int k = k_next + thread * parts;
                bool hit = false;
                if (k < last) {
                    const float4 a = __ldg(recs + 4 * (size_t)k);
                    hit = fabsf(a.x * cx + a.y * cy + a.z * cz) <= fabsf(a.x) * hx + fabsf(a.y) * hy + fabsf(a.z) * hz + kBrickSlack;
                    if (hit) {
                        const float2 e = __ldg(reinterpret_cast<const float2*>(recs + 4 * (size_t)k + 1));
                        hit = a.w * cx + e.x * cy + e.y * cz + fabsf(a.w) * hx + fabsf(e.x) * hy + fabsf(e.y) * hz >= -kBrickSlack;
                    }
                }
                const unsigned m = __ballot_sync(kFull, hit);
                int pos = nhits;
                if (kAlone) {
                    nhits += __popc(m);
                } else {
                    if (lane == 0 && m) pos = atomicAdd(&sb.nhits, __popc(m));
                    pos = __shfl_sync(kFull, pos, 0);
                }
                if (hit) sb.hits[pos + __popc(m & upto) - 1] = k;
            }
            if (kAlone) {
                __syncwarp();
            } else {
                __syncthreads();
                nhits = sb.nhits;
                __syncthreads();
            }
        } while (k_next < last && nhits + kThreads <= BLOCK::kHits);
        for (int h_next = 0;; h_next += grab) {
            int h = h_next;
            if (!kAlone) {
                if (lane == 0) h = atomicAdd(&sb.next, grab);
                h = __shfl_sync(kFull, h, 0);
            }
            if (h >= nhits) break;
            const int slices = min(grab, nhits - h);
            int row_count = 0, k_lo = 0;
            if (lane < slices) {
                const int slice = sb.hits[h + lane];
                const float4 e = __ldg(recs + 4 * (size_t)slice + 1), f = __ldg(recs + 4 * (size_t)slice + 2), v = __ldg(recs + 4 * (size_t)slice + 3);
                const float2 s = g.has_shift ? __ldg(shifts + slice) : make_float2(0.f, 0.f);
                sw.slice[lane] = slice;
                sw.slots[lane][0] = make_float4(e.z, e.w, f.x, f.y);
                sw.slots[lane][1] = make_float4(f.z, f.w, s.x, s.y);
                const float mid = v.x * cx + v.y * cy + v.z * cz;
                const float reach = fabsf(v.x) * (hx + kBrickSlack) + fabsf(v.y) * (hy + kBrickSlack) + fabsf(v.z) * (hz + kBrickSlack);
                k_lo = max((int)ceilf((mid - reach) * inv_os), 1 - g.N / 2);
                row_count = max(1, min((int)floorf((mid + reach) * inv_os), g.N / 2) - k_lo + 1);
            }
            int row_incl = row_count;
#pragma unroll
            for (int o = 1; o < kBrickSlots; o <<= 1) {
                const int up = __shfl_up_sync(kFull, row_incl, o);
                if (lane >= o) row_incl += up;
            }
            const int row_start = row_incl - row_count, rows = __shfl_sync(kFull, row_incl, kBrickSlots - 1);
            const int kr_start = k_lo - row_start;
            __syncwarp();
            int nseg = 0, row0 = 0, slots_before = 0;
            while (true) {
            while (row0 < rows && nseg < 32) {
                const unsigned starts = __reduce_or_sync(kFull, (lane < slices && row_start >= row0 && row_start < row0 + 32) ? 1u << (row_start - row0) : 0u);
                const int slot = slots_before + __popc(starts & upto) - 1;
                slots_before += __popc(starts);
                const int kr = row0 + lane + __shfl_sync(kFull, kr_start, slot);
                const float krf = (float)kr;
                const float4 ra = sw.slots[slot][0], rb = sw.slots[slot][1];
                const float room = g.cutoff_sq - krf * krf;
                int ja_i = 0, len = 0;
                if (row0 + lane < rows && room >= 0.f && kr <= g.N / 2) {       // (a slice without rows here still counts one)
                    float ja = 0.f, jb = fminf((float)(g.Nh - 1), sqrtf(room) + 0.01f);
                    auto clip = [&](float a, float b, float lo, float n) {
                        a *= osf;
                        b *= osf * krf;
                        if (fabsf(a) < 1e-5f) {
                            if (b < lo - kBrickSlack || b > lo + n + kBrickSlack) jb = -1.f;
                        } else {
                            const float ia = __fdividef(1.f, a);
                            const float x0 = (lo - kBrickSlack - b) * ia, x1 = (lo + n + kBrickSlack - b) * ia;
                            ja = fmaxf(ja, fminf(x0, x1));
                            jb = fminf(jb, fmaxf(x0, x1));
                        }
                    };
                    clip(ra.x, ra.w, (float)X0, (float)D::x);
                    clip(ra.y, rb.x, (float)Y0, (float)D::y);
                    if (D::kDim == 3) clip(ra.z, rb.y, (float)Z0, (float)D::z);
                    ja_i = (int)ceilf(ja);
                    len = jb >= ja ? (int)floorf(jb) - ja_i + 1 : 0;
                }
                const unsigned have = __ballot_sync(kFull, len > 0);
                if (len > 0) sw.segs[nseg + __popc(have & upto) - 1] = make_uint2((unsigned)slot << 16 | ((unsigned)kr & 0xffffu), (unsigned)ja_i << 16 | (unsigned)len);
                nseg += __popc(have);
                row0 += 32;
            }
            if (nseg == 0) break;
            __syncwarp();
            const int take = min(nseg, 32);
            const uint2 seg = lane < take ? sw.segs[lane] : make_uint2(0u, 0u);
            const int len = (int)(seg.y & 0xffffu);
            int incl = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += up;
            }
            const int total = __shfl_sync(kFull, incl, 31), start = incl - len;
            const int ja_start = (int)(seg.y >> 16) - start;
            int before = 0;                                           // segments that start before the window
            for (int k0 = 0; k0 < total; k0 += 32) {
                const unsigned bit = (len > 0 && start >= k0 && start < k0 + 32) ? 1u << (start - k0) : 0u;
                const unsigned starts = __reduce_or_sync(kFull, bit);
                const int src = before + __popc(starts & upto) - 1;
                before += __popc(starts);
                const unsigned sk = __shfl_sync(kFull, seg.x, src);
                const int j = k0 + lane + __shfl_sync(kFull, ja_start, src);
                const int kr = (int)(short)(sk & 0xffffu), slot = (int)(sk >> 16);
                const float4 ra = sw.slots[slot][0], rb = sw.slots[slot][1];
                Pixel px;
                px.kr = (float)kr;
                px.kc = (float)j;
                if (g.os_is_float) {
                    px.sc = mul_rn(px.kc, g.os_f);
                    px.sr = mul_rn(px.kr, g.os_f);
                } else {
                    px.sc = (float)((double)px.kc * g.os);
                    px.sr = (float)((double)px.kr * g.os);
                }
                px.c = add_rn(mul_rn(ra.x, px.sc), mul_rn(ra.w, px.sr));
                px.r = add_rn(mul_rn(ra.y, px.sc), mul_rn(rb.x, px.sr));
                px.d = D::kDim == 3 ? add_rn(mul_rn(ra.z, px.sc), mul_rn(rb.y, px.sr)) : 0.f;
                int lx = (int)floorf(px.c) - X0, ly = (int)floorf(px.r) - Y0, lz = D::kDim == 3 ? (int)floorf(px.d) - Z0 : 0;
                const float rad = add_rn(mul_rn(px.kr, px.kr), mul_rn(px.kc, px.kc));
                const bool active = k0 + lane < total && (unsigned)lx < (unsigned)D::x && (unsigned)ly < (unsigned)D::y &&
                                    (D::kDim == 2 || (unsigned)lz < (unsigned)D::z) && !(rad > g.cutoff_sq);
                if (!active) lx = ly = lz = 0;
                body(active, slot, kr < 0 ? kr + g.N : kr, j, px, lx, ly, lz);
            }
            nseg -= take;
            const uint2 rest = lane < nseg ? sw.segs[take + lane] : make_uint2(0u, 0u);
            __syncwarp();
            if (lane < nseg) sw.segs[lane] = rest;
            __syncwarp();
            }
        }
    }
}

// A pixel's saved derivatives: a record in 3D, two planes in 2D.
template <int DIM>
__device__ __forceinline__ void brick_save(const SliceGeom& g, float2* __restrict__ derivs, size_t pix, float2 gc, float2 gr, float2 gd, float2 v) {
    if (DIM == 3) {
        store_record(derivs + 4 * pix, gc, gr, gd, v);
    } else {
        __stcg(derivs + pix, gc);
        __stcg(derivs + (size_t)g.BP * (size_t)g.slice_pixels + pix, gr);
    }
}

// What the bricks leave of a slice: zeros outside the cutoff, or -- when its matrix is nearly singular or stretches
// beyond the shells -- the whole slice, by the plain gather.
template <int DIM, bool CUBIC, bool SAVE>
__device__ __forceinline__ void brick_rest(const SliceGeom& g, const BrickWork& ws, int k, const float2* __restrict__ rec, const float* __restrict__ rot,
                                           const float* __restrict__ shifts, float2* __restrict__ out, float2* __restrict__ derivs) {
    const int b = k / g.P, p = k - b * g.P;
    const float* rm = pose_rot<DIM>(g, rot, b, p);
    const size_t base = (size_t)k * (size_t)g.slice_pixels;
    if (brick_has_slice(ws, k)) {
        const int n = __ldg(ws.header + 3);
        for (int q = threadIdx.x; q < n; q += kBlockThreads) __stcs(out + (base + (size_t)__ldg(ws.outside + q)), make_float2(0.f, 0.f));
        return;
    }
    for (int tile = 0; tile < g.tiles_i * g.tiles_j; ++tile) {
        int i, j;
        tile_pixel(g, tile, i, j);
        Pixel px;
        px.c = px.r = px.d = 0.f;
        const bool in_image = i < g.N && j < g.Nh;
        const bool valid = in_image && pixel_setup<DIM>(g, rm, i, j, px);
        float2 v, gc, gr, gd;
        interpolate_any<DIM, CUBIC, SAVE>(g, rec + (size_t)b * g.vol_elems, px, valid, v, gc, gr, gd);
        if (!in_image) continue;
        float2 ph = make_float2(1.f, 0.f);
        if (valid && g.has_shift) {
            const float* s = pose_shift(g, shifts, b, p);
            ph = phase_ramp(g, px, __ldg(s), __ldg(s + 1));
            v = cmul(v, ph);
        }
        const size_t pix = base + (size_t)(i * g.Nh + j);
        __stcs(out + pix, v);
        if (SAVE && valid) brick_save<DIM>(g, derivs, pix, g.has_shift ? cmul(gc, ph) : gc, g.has_shift ? cmul(gr, ph) : gr, DIM == 3 && g.has_shift ? cmul(gd, ph) : gd, v);
    }
}

using GatherBlock = BrickBlock<kWarps, 1024>;

// Forward projection (SAVE: with the derivatives of project_forw_saving_kernel, 3D as records).
template <int DIM, bool CUBIC, bool SAVE>
__global__ void __launch_bounds__(kBlockThreads, CUBIC ? 3 : 4)
brick_forw_kernel(const float2* __restrict__ rec, const float* __restrict__ rot, const float* __restrict__ shifts,
                  float2* __restrict__ out, float2* __restrict__ derivs, BrickWork ws, const SliceGeom g, const BrickPlan pl) {
    extern __shared__ __align__(16) unsigned char dyn[];
    float2* sm = reinterpret_cast<float2*>(dyn);
    GatherBlock& sb = *reinterpret_cast<GatherBlock*>(dyn + sizeof(float2) * BrickShape<DIM, CUBIC>::kVoxels);
    const int items = brick_items(ws);
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) sb.item = atomicAdd(ws.header + 2, 1);
        __syncthreads();
        const int item = sb.item;
        if (item >= items) return;
        // beside its brick an item does its share of the slices' rest, whose stores overlap the brick's staging
        for (int k = (int)((long long)g.BP * item / items), k_end = (int)((long long)g.BP * (item + 1) / items); k < k_end; ++k)
            brick_rest<DIM, CUBIC, SAVE>(g, ws, k, rec, rot, shifts, out, derivs);
        const int4 it = brick_item(ws, pl, item);
        const int X0 = pl.lo[0] + (it.x & 1023) * GatherBrick<DIM, CUBIC>::x, Y0 = pl.lo[1] + ((it.x >> 10) & 1023) * GatherBrick<DIM, CUBIC>::y, Z0 = pl.lo[2] + (it.x >> 20) * GatherBrick<DIM, CUBIC>::z;
        brick_stage<DIM, CUBIC>(g, rec + (size_t)it.y * g.vol_elems, sm, X0, Y0, Z0);
        const BrickWarp& sw = sb.warp[threadIdx.x >> 5];
        brick_walk<GatherBrick<DIM, CUBIC>>(g, ws.recs, ws.shifts, sb, X0, Y0, Z0, it.z, it.w, 0, 1,
                   [&](bool active, int slot, int i, int j, const Pixel& px, int lx, int ly, int lz) {
            float2 v, gc, gr, gd;
            brick_gather<DIM, CUBIC, SAVE>(sm, lx, ly, lz, px.c - floorf(px.c), px.r - floorf(px.r), DIM == 3 ? px.d - floorf(px.d) : 0.f, v, gc, gr, gd);
            if (!active) return;
            if (g.has_shift) {
                const float4 rc = sw.slots[slot][1];
                const float2 ph = phase_ramp(g, px, rc.z, rc.w);
                v = cmul(v, ph);
                if (SAVE) {
                    gc = cmul(gc, ph);
                    gr = cmul(gr, ph);
                    if (DIM == 3) gd = cmul(gd, ph);
                }
            }
            const size_t pix = (size_t)sw.slice[slot] * (size_t)g.slice_pixels + (size_t)(i * g.Nh + j);
            __stcg(out + pix, v);
            if (SAVE) brick_save<DIM>(g, derivs, pix, gc, gr, gd, v);
        });
    }
}

}  // namespace b200proj
