// Cell-sorted scatters (fp32): back-projection, and the gradient of the projection with respect to the reconstruction,
// from pixel lists (pixel_lists.cuh).  A work item is a brick of 512 cells and a run of its list.  A block reads the run in
// batches into shared memory and chains the pixels of each cell; then a thread takes a cell's chain and adds its pixels up
// in registers -- all pixels of a cell have the same taps --, so that no two threads ever add to the same place and
// a tap costs one fused multiply-add instead of a reduction sent to L2.
//
// What cannot be added up this way without changing results -- a pixel whose value or weight is infinite or NaN, of
// which the taps of weight zero must see nothing -- is sent to memory tap by tap.
#pragma once

#include "pixel_lists.cuh"

namespace b200proj {

// Where a scatter's sums go: 16-byte (re, im, weight, 0) voxels, or a complex volume and one of weights.
template <bool WEIGHTS, bool INTERLEAVED>
struct ScatterTarget {
    float2* vol;
    float* wvol;
    float4* accum;
    __device__ __forceinline__ void add(long long off, float re, float im, float w) const {
        if (INTERLEAVED) {
            red_add_v4(accum + off, re, im, w, 0.f);
        } else {
            red_add_v2(vol + off, re, im);
            if (WEIGHTS) red_add(wvol + off, w);
        }
    }
};

// One voxel's sum by the scatter's rules: Friedel mirror with conjugation, taps outside the stored half dropped, DUP: the
// conjugate also to the Friedel partner of a voxel on the c == 0 plane.
template <int DIM, bool DUP, typename Target>
__device__ __forceinline__ void scatter_voxel(const SliceGeom& g, const Target& to, long long item, int c, int r, int d, float re, float im, float w) {
    bool m;
    c = scatter_col(g, c, m);
    r = scatter_line(g, r, m);
    d = DIM == 3 ? scatter_line(g, d, m) : 0;
    if (c < 0 || r < 0 || d < 0) return;
    if (m) im = -im;
    to.add(item + ((d * g.R + r) * g.Rh + c), re, im, w);
    if (DUP && c == 0) {
        const int r2 = r == 0 ? 0 : g.R - r, d2 = d == 0 ? 0 : g.R - d;
        if (r2 != r || d2 != d) to.add(item + (d2 * g.R + r2) * g.Rh, re, -im, w);
    }
}

__device__ __forceinline__ bool finite_values(float2 v, float w) { return fabsf(v.x) + fabsf(v.y) + fabsf(w) < __int_as_float(0x7f800000); }

// A pixel by itself, tap by tap; taps of weight zero are skipped.
template <int DIM, bool CUBIC, bool DUP, typename Target>
__device__ __noinline__ void scatter_alone(const SliceGeom& g, const Target& to, long long item, float c, float r, float d, float2 v, float w) {
    constexpr int T = CUBIC ? 4 : 2;
    AxisWeights<float, T> ac, ar, ad;
    axis_weights<T, false>(c, ac);
    axis_weights<T, false>(r, ar);
    if (DIM == 3) axis_weights<T, false>(d, ad);
#pragma unroll 1
    for (int t = 0; t < (DIM == 3 ? T * T * T : T * T); ++t) {
        const int x = t % T, y = t / T % T, z = DIM == 3 ? t / (T * T) : 0;
        const float fz = DIM == 3 ? (z == 0 ? ad.w[0] : z == 1 ? ad.w[1] : z == 2 ? ad.w[T - 2] : ad.w[T - 1]) : 1.f;
        const float fy = y == 0 ? ar.w[0] : y == 1 ? ar.w[1] : y == 2 ? ar.w[T - 2] : ar.w[T - 1];
        const float fx = x == 0 ? ac.w[0] : x == 1 ? ac.w[1] : x == 2 ? ac.w[T - 2] : ac.w[T - 1];
        if (fz == 0.f || fy == 0.f || fx == 0.f) continue;          // (each by itself: beside a NaN the product is one)
        const float f = fz * fy * fx;
        scatter_voxel<DIM, DUP>(g, to, item, ac.base + x, ar.base + y, DIM == 3 ? ad.base + z : 0, v.x * f, v.y * f, w * fabsf(f));
    }
}

// ---- reading a batch -----------------------------------------------------------------------------------------
template <int DIM>
struct CellDims {
    using L = ListBrick<DIM>;
    static constexpr int kLogX = L::kLogX, kLogY = L::kLogY, kLogZ = L::kLogZ;
    static constexpr int kX = 1 << L::kLogX, kY = 1 << L::kLogY, kZ = 1 << L::kLogZ, kCells = kX * kY * kZ;
};
struct CellBrick {
    int x, y, z, b;         // first cell (signed coordinates), batch item
};
template <typename D>
__device__ __forceinline__ CellBrick cell_brick(const ListPlan& pl, int brick) {
    CellBrick k;
    const int row = brick / pl.n[0], plane = row / pl.n[1];
    k.x = pl.lo[0] + (brick - row * pl.n[0]) * D::kX;
    k.y = pl.lo[1] + (row - plane * pl.n[1]) * D::kY;
    k.b = plane / pl.n[2];
    k.z = pl.lo[2] + (plane - k.b * pl.n[2]) * D::kZ;
    return k;
}

struct CellEntry {
    int slice;
    unsigned row, column;
    size_t pix;
};
__device__ __forceinline__ CellEntry cell_entry(const SliceGeom& g, const ListPlan& pl, unsigned e) {
    CellEntry k;
    k.column = e & ((1u << pl.bits_j) - 1u);
    k.row = (e >> pl.bits_j) & ((1u << pl.bits_i) - 1u);
    k.slice = pl.first + (int)(e >> (pl.bits_i + pl.bits_j));
    const int kr = (int)k.row - (g.N / 2 - 1), i = kr < 0 ? kr + g.N : kr;
    k.pix = (size_t)k.slice * (size_t)g.slice_pixels + (size_t)(i * g.Nh + (int)k.column);
    return k;
}

// What the lists leave of a scatter, a block per slice: slices that are not listed, and pixels whose value or weight is not
// finite (the taps of weight zero must see nothing of them).  Nearly always there is nothing to do.
template <int DIM, bool CUBIC, bool WEIGHTS, bool DUP, typename Target>
__global__ void __launch_bounds__(256)
scatter_rest_kernel(const float2* __restrict__ proj, const float* __restrict__ weights, const float* __restrict__ rot, const float* __restrict__ shifts,
                    const Target to, const ListWork ws, const SliceGeom g, const ListPlan pl) {
    if (Gate::crowded(ws.header, pl.crowd)) return;
    const bool odd = __ldg(ws.header + 5) != 0;
    if (!odd && __ldg(ws.header + 4) == 0) return;
    for (int k = pl.first + (int)blockIdx.x; k < pl.first + pl.slices; k += (int)gridDim.x) {
        const bool all = isnan(__ldg(&ws.poses[2 * (size_t)k].x));
        if (!all && !odd) continue;
        const int b = k / g.P, p = k - b * g.P;
        for (int t = (int)threadIdx.x; t < g.slice_pixels; t += 256) {
            const int i = t / g.Nh, j = t - i * g.Nh;
            const size_t pix = (size_t)k * (size_t)g.slice_pixels + (size_t)t;
            Pixel px;
            if ((j == 0 && i >= g.N / 2) || !pixel_setup<DIM>(g, pose_rot<DIM>(g, rot, b, p), i, j, px)) continue;
            float2 v = __ldg(proj + pix);
            const float w = WEIGHTS ? __ldg(weights + pix) : 0.f;
            if (g.has_shift) {              // of listed slices as where the sums are formed, so that both find the same pixels finite
                const float dot = add_rn(mul_rn(px.kr, __ldg(pose_shift(g, shifts, b, p))), mul_rn(px.kc, __ldg(pose_shift(g, shifts, b, p) + 1)));
                v = cmul_conj(v, all ? phase_of_dot(g, dot) : list_phase(g, dot));
            }
            if (all || !finite_values(v, w)) scatter_alone<DIM, CUBIC, DUP>(g, to, (long long)b * g.vol_elems, px.c, px.r, px.d, v, w);
        }
    }
}

// ---- reading batches ahead -----------------------------------------------------------------------------------
// The batches of a block, in shared memory.  It takes items from a ticket counter (in turn, blocks would drift apart, and with
// them the neighbours that read the same sectors), each in batches of nearly equal size.  Thread 0 keeps the queue two
// batches ahead, and fetches the item after those and the ticket after that before they are needed.
struct CellQueue {
    int4 batch[4];          // {brick, first entry, entries (0: no more), whether it ends its item}
    int4 ahead;             // the next item {brick, first entry, entries}
    int brick, first, left, size, items;
};
__device__ __forceinline__ void queue_push(CellQueue& q, const ListWork& ws, int s, int most, int& ticket) {
    if (q.left == 0) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        const int4 it = q.ahead;
        if (it.z == 0) {
            q.batch[s & 3] = make_int4(0, 0, 0, 0);
            return;
        }
        const int batches = (it.z + most - 1) / most;
        q.brick = it.x;
        q.first = it.y;
        q.left = it.z;
        q.size = (it.z + batches - 1) / batches;
        if (ticket < q.items) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(&q.ahead)), "l"(ws.items + ticket) : "memory");
        else q.ahead = make_int4(0, 0, 0, 0);
        ticket = 2 * (int)gridDim.x + atomicAdd(ws.header + 2, 1);
    }
    const int n = min(q.size, q.left);
    q.batch[s & 3] = make_int4(q.brick, q.first, n, n == q.left);
    q.first += n;
    q.left -= n;
}
// By all threads; the first two batches are in the queue after the next barrier.
__device__ __forceinline__ void queue_start(CellQueue& q, const ListWork& ws, int most, int& ticket) {
    if (threadIdx.x != 0) return;
    q.items = __ldg(ws.header + 1);
    q.left = 0;
    q.ahead = (int)blockIdx.x < q.items ? __ldg(ws.items + blockIdx.x) : make_int4(0, 0, 0, 0);
    ticket = (int)(blockIdx.x + gridDim.x);
    queue_push(q, ws, 0, most, ticket);
    queue_push(q, ws, 1, most, ticket);
}

template <int RUN, int THREADS>
__device__ __forceinline__ void cell_entries(const ListWork& ws, int first, int n, unsigned (&e)[RUN]) {
#pragma unroll
    for (int q = 0; q < RUN; ++q) {
        const int t = q * THREADS + (int)threadIdx.x;
        e[q] = t < n ? __ldcs(ws.list + first + t) : 0u;
    }
}
// The batch's pixels: place(at, cell, sample, value, weight) for each, values with their shift phase.  Returns whether some value is
// not finite (it counts as zero here, see scatter_rest_kernel).
template <int DIM, typename D, int RUN, int THREADS, bool WEIGHTS, typename Place>
__device__ __forceinline__ bool cell_place(const SliceGeom& g, const ListPlan& pl, const ListWork& ws, const float2* __restrict__ proj, const float* __restrict__ weights,
                                           int n, const unsigned (&e)[RUN], Place place) {
    bool odd = false;
    float2 v[RUN];
    float w[RUN];
#pragma unroll
    for (int q = 0; q < RUN; ++q) {
        const bool mine = q * THREADS + (int)threadIdx.x < n;
        const size_t pix = cell_entry(g, pl, e[q]).pix;
        v[q] = mine ? __ldg(proj + pix) : make_float2(0.f, 0.f);
        w[q] = WEIGHTS && mine ? __ldg(weights + pix) : 0.f;
    }
#pragma unroll
    for (int q = 0; q < RUN; ++q) {
        const int t = q * THREADS + (int)threadIdx.x;
        const unsigned column = e[q] & ((1u << pl.bits_j) - 1u), row = (e[q] >> pl.bits_j) & ((1u << pl.bits_i) - 1u);
        const float4* pose = ws.poses + 2 * (size_t)(pl.first + (int)(e[q] >> (pl.bits_i + pl.bits_j)));
        const float4 ra = __ldg(pose), rb = __ldg(pose + 1);
        const ListSample s = list_sample<DIM>(g, pl, ra, rb, row, column);
        if (g.has_shift) v[q] = cmul_conj(v[q], list_phase(g, add_rn(mul_rn(s.kr, rb.z), mul_rn(s.kc, rb.w))));
        if (s.folded) v[q].y = -v[q].y;
        const bool finite = finite_values(v[q], w[q]);
        odd |= !finite && t < n;
        if (t < n && finite)
            place(t, (s.x & (D::kX - 1)) | (s.y & (D::kY - 1)) << D::kLogX | (DIM == 3 ? (s.z & (D::kZ - 1)) << (D::kLogX + D::kLogY) : 0), s, v[q], w[q]);
    }
    return odd;
}

// The sums of an item's voxels, in shared memory (rows of ROW), to the volume.
template <int DIM, bool WEIGHTS, bool DUP, int SX, int SY, int SZ, int ROW, int THREADS, typename Target>
__device__ __forceinline__ void cell_flush(const SliceGeom& g, const Target& to, const CellBrick& brick, int halo, float2* v, float* w) {
    for (int t = (int)threadIdx.x; t < SX * SY * SZ; t += THREADS) {
        const int row = t / SX, x = t - row * SX, z = row / SY, y = row - z * SY, at = row * ROW + x;
        const float2 u = v[at];
        const float f = WEIGHTS ? w[at] : 0.f;
        if (u.x == 0.f && u.y == 0.f && f == 0.f) continue;
        scatter_voxel<DIM, DUP>(g, to, (long long)brick.b * g.vol_elems, brick.x - halo + x, brick.y - halo + y, brick.z - halo + z, u.x, u.y, f);
    }
}

// ---- a thread per cell: linear taps, and cubic ones in 2D --------------------------------------------------------------
// The thread keeps the sums of its cell's taps in registers over all batches of an item.
template <int DIM, bool CUBIC, bool WEIGHTS>
struct CellSums {
    using D = CellDims<DIM>;
    // pixels of a thread in a batch: more keep more lanes busy in the chains, fewer leave more of L1.  2D, 3,000 slices of 128 x 65, cubic
    // and weighted: 4 299 us, 6 288, 8 256; without weights 4 287, 5 281, 8 340 (8 x 500 slices); linear 4 427, 5 440, 8 743; 3D linear 4 4.16 ms, 5 4.56
    static constexpr int kThreads = D::kCells, kRun = DIM == 3 || !CUBIC ? 4 : WEIGHTS ? 8 : 5, kBatch = kThreads * kRun;
    static constexpr int kBlocks = DIM == 3 ? 2 : !CUBIC ? 4 : WEIGHTS ? 2 : 3;
    static constexpr int T = CUBIC ? 4 : 2, kHalo = CUBIC ? 1 : 0, kRows = DIM == 3 ? T * T : T;
    static constexpr int kSX = D::kX + T - 1, kSY = D::kY + T - 1, kSZ = DIM == 3 ? D::kZ + T - 1 : 1;
    static constexpr int kRow = DIM == 3 ? 24 : kSX;        // 3D: the rows of a warp's cells meet different banks
    static constexpr int kVoxels = kRow * kSY * kSZ;
    struct Batch {
        float4 a[kBatch];                   // fractions, weight
        float2 v[kBatch];
        short next[kBatch];                 // place of the cell's next pixel
    };
    struct Sums {
        float2 v[kVoxels];
        float w[WEIGHTS ? kVoxels : 4];
    };
    struct Shared {
        union {
            Batch batch;
            Sums sums;
        };
        int head[kThreads];
        CellQueue queue;
    };
};
constexpr int kChainEnd = -1;

template <int DIM, bool CUBIC, bool WEIGHTS, bool DUP, bool INTERLEAVED>
__global__ void __launch_bounds__(CellSums<DIM, CUBIC, WEIGHTS>::kThreads, CellSums<DIM, CUBIC, WEIGHTS>::kBlocks)
cell_sums_kernel(const float2* __restrict__ proj, const float* __restrict__ weights, const ScatterTarget<WEIGHTS, INTERLEAVED> to, const ListWork ws,
                 const SliceGeom g, const ListPlan pl) {
    if (Gate::crowded(ws.header, pl.crowd)) return;
    using C = CellSums<DIM, CUBIC, WEIGHTS>;
    using D = typename C::D;
    using u64 = unsigned long long;
    extern __shared__ __align__(16) unsigned char dyn[];
    typename C::Shared& sh = *reinterpret_cast<typename C::Shared*>(dyn);
    constexpr int T = C::T;
    const int tid = threadIdx.x, cx = tid & (D::kX - 1), cy = (tid >> D::kLogX) & (D::kY - 1), cz = tid >> (D::kLogX + D::kLogY);
    int ticket;
    queue_start(sh.queue, ws, C::kBatch, ticket);
    sh.head[tid] = kChainEnd;
    __syncthreads();
    u64 acc[C::kRows][T];
    float wacc[C::kRows][T];
#pragma unroll
    for (int r = 0; r < C::kRows; ++r)
#pragma unroll
        for (int x = 0; x < T; ++x) {
            acc[r][x] = 0ull;
            wacc[r][x] = 0.f;
        }
    unsigned e[C::kRun];
    cell_entries<C::kRun, C::kThreads>(ws, sh.queue.batch[0].y, sh.queue.batch[0].z, e);
    bool odd = false;
    for (int s = 0;; ++s) {
        const int n = sh.queue.batch[s & 3].z;
        if (n == 0) break;
        odd |= cell_place<DIM, D, C::kRun, C::kThreads, WEIGHTS>(g, pl, ws, proj, weights, n, e, [&](int t, int cell, const ListSample& s, float2 v, float w) {
            sh.batch.a[t] = make_float4(s.fc, s.fr, s.fd, w);
            sh.batch.v[t] = v;
            sh.batch.next[t] = (short)atomicExch(&sh.head[cell], t);
        });
        cell_entries<C::kRun, C::kThreads>(ws, sh.queue.batch[(s + 1) & 3].y, sh.queue.batch[(s + 1) & 3].z, e);
        __syncthreads();
        if (tid == 0) queue_push(sh.queue, ws, s + 2, C::kBatch, ticket);
        int p = sh.head[tid];
        sh.head[tid] = kChainEnd;
        while (p != kChainEnd) {
            const float4 a = sh.batch.a[p];
            const float2 u = sh.batch.v[p];
            const float w = a.w;
            p = sh.batch.next[p];
            const u64 u2 = pack2(u.x, u.y);
            float wx[T], wy[T];
            if constexpr (CUBIC) {
                cubic_weights(a.x, wx);
                cubic_weights(a.y, wy);
            } else {
                wx[0] = 1.f - a.x;
                wx[1] = a.x;
                wy[0] = 1.f - a.y;
                wy[1] = a.y;
            }
#pragma unroll
            for (int r = 0; r < C::kRows; ++r) {
                const float f = DIM == 3 ? wy[r % T] * (r / T ? a.z : 1.f - a.z) : wy[r];
                const u64 q2 = fmul2(u2, pack2(f, f));
                const float fw = w * fabsf(f);
#pragma unroll
                for (int x = 0; x < T; ++x) {
                    acc[r][x] = fma2(q2, pack2(wx[x], wx[x]), acc[r][x]);
                    if (WEIGHTS) wacc[r][x] = fmaf(fw, fabsf(wx[x]), wacc[r][x]);
                }
            }
        }
        __syncthreads();
        if (sh.queue.batch[s & 3].w) {
            // The cells' sums into those of the brick's voxels, row by row of the footprint: the warps hold different rows of
            // cells, and within a warp different cells add to different voxels at each tap.
            for (int t = tid; t < C::kVoxels; t += C::kThreads) {
                sh.sums.v[t] = make_float2(0.f, 0.f);
                if (WEIGHTS) sh.sums.w[t] = 0.f;
            }
            const int to_row = (cz * C::kSY + cy) * C::kRow + cx;
#pragma unroll
            for (int r = 0; r < C::kRows; ++r) {
                __syncthreads();
#pragma unroll
                for (int x = 0; x < T; ++x) {
                    const int t = to_row + x + (r % T) * C::kRow + (r / T) * (C::kRow * C::kSY);
                    float re, im;
                    unpack2(acc[r][x], re, im);
                    acc[r][x] = 0ull;
                    const float2 u = sh.sums.v[t];
                    sh.sums.v[t] = make_float2(u.x + re, u.y + im);
                    if (WEIGHTS) {
                        sh.sums.w[t] += wacc[r][x];
                        wacc[r][x] = 0.f;
                    }
                    __syncwarp();
                }
            }
            __syncthreads();
            cell_flush<DIM, WEIGHTS, DUP, C::kSX, C::kSY, C::kSZ, C::kRow, C::kThreads>(g, to, cell_brick<D>(pl, sh.queue.batch[s & 3].x), C::kHalo, sh.sums.v, sh.sums.w);
            __syncthreads();
        }
    }
    if (odd) ws.header[5] = 1;
}

// ---- cubic taps in 3D ---------------------------------------------------------------------------------------
// A cell has 64 taps: kSplit threads share it, each with some of the planes of its footprint.  A warp has a layer of the
// brick, 8 x 8 cells, which it takes 16 (8) at a time, and sums of its own for the four planes that they add to; so
// the warps do not wait for one another between the placement of a batch and its end.  Within a warp all cells add at the same
// tap of their footprints: different voxels.
// The lanes of a round wait for the longest chain among its cells.  So the cells of a layer are dealt out by the
// bank of their first voxel, those of a bank from the longest chain to the shortest: the chains of a round are of
// similar length, and its cells of different banks (in the order of the rows: 3.86 instead of 3.69 ms, weighted, 2,501 slices
// of 90 x 46, 599 instead of 544 us).  (One set of sums for the block, with barriers between the rows of the
// footprints: 4.28 instead of 3.94 ms for 4,096 slices of 256 x 129 into a box-512 volume.)
template <bool WEIGHTS>
struct CubicSums {
    using D = CellDims<3>;
    static constexpr int kSplit = WEIGHTS ? 4 : 2, kPlanes = 4 / kSplit, kThreads = 32 * D::kZ, kRun = WEIGHTS ? 7 : 8, kBatch = kThreads * kRun, kBlocks = 2;
    static constexpr int kWarpCells = 32 / kSplit, kRounds = D::kX * D::kY / kWarpCells;
    // rows of 12 voxels and, for planes side by side in a warp, planes 8 banks apart: every bank has as many of a layer's cells
    static constexpr int kSX = D::kX + 3, kSY = D::kY + 3, kSZ = D::kZ + 3, kRow = 12, kPlane = 136;
    static_assert(kPlane >= kRow * kSY && kRow % 8 == 4 && kPlane % 16 == 8, "banks");
    struct Shared {
        float4 a[kBatch];                   // fractions, place of the cell's next pixel
        float2 v[kBatch];
        float w[WEIGHTS ? kBatch : 4];
        float2 sum[D::kZ][4 * kPlane];
        float wsum[WEIGHTS ? D::kZ : 1][WEIGHTS ? 4 * kPlane : 4];
        int head[D::kCells], count[D::kCells];
        unsigned char order[D::kZ][D::kX * D::kY];      // cells of a layer, round by round
        CellQueue queue;
    };
};

template <bool WEIGHTS, bool DUP, bool INTERLEAVED>
__global__ void __launch_bounds__(CubicSums<WEIGHTS>::kThreads, CubicSums<WEIGHTS>::kBlocks)
cell_cubic_sums_kernel(const float2* __restrict__ proj, const float* __restrict__ weights, const ScatterTarget<WEIGHTS, INTERLEAVED> to, const ListWork ws,
                       const SliceGeom g, const ListPlan pl) {
    if (Gate::crowded(ws.header, pl.crowd)) return;
    using C = CubicSums<WEIGHTS>;
    using D = typename C::D;
    using u64 = unsigned long long;
    extern __shared__ __align__(16) unsigned char dyn[];
    typename C::Shared& sh = *reinterpret_cast<typename C::Shared*>(dyn);
    const int tid = threadIdx.x, lane = tid & 31, cz = tid >> 5;
    const int part = lane / C::kWarpCells;              // lanes of the same cell are kWarpCells apart
    float2* sum = sh.sum[cz];
    float* wsum = sh.wsum[WEIGHTS ? cz : 0];
    int ticket;
    queue_start(sh.queue, ws, C::kBatch, ticket);
    for (int t = tid; t < D::kCells; t += C::kThreads) {
        sh.head[t] = kChainEnd;
        sh.count[t] = 0;
    }
    for (int t = tid; t < D::kZ * 4 * C::kPlane; t += C::kThreads) {
        sh.sum[0][t] = make_float2(0.f, 0.f);
        if (WEIGHTS) sh.wsum[0][t] = 0.f;
    }
    __syncthreads();
    unsigned e[C::kRun];
    cell_entries<C::kRun, C::kThreads>(ws, sh.queue.batch[0].y, sh.queue.batch[0].z, e);
    bool odd = false;
    for (int s = 0;; ++s) {
        const int n = sh.queue.batch[s & 3].z;
        if (n == 0) break;
        odd |= cell_place<3, D, C::kRun, C::kThreads, WEIGHTS>(g, pl, ws, proj, weights, n, e, [&](int t, int cell, const ListSample& at, float2 v, float w) {
            sh.a[t] = make_float4(at.fc, at.fr, at.fd, __int_as_float(atomicExch(&sh.head[cell], t)));
            sh.v[t] = v;
            if (WEIGHTS) sh.w[t] = w;
            atomicAdd(&sh.count[cell], 1);
        });
        cell_entries<C::kRun, C::kThreads>(ws, sh.queue.batch[(s + 1) & 3].y, sh.queue.batch[(s + 1) & 3].z, e);
        __syncthreads();
        if (tid == 0) queue_push(sh.queue, ws, s + 2, C::kBatch, ticket);
        __syncwarp();
        {
            // the cells of this lane's bank, longest chain first
            int keys[C::kRounds];
#pragma unroll
            for (int k = 0; k < C::kRounds; ++k) {
                // rows of a bank: kSplit 4: all (cx + 4 cy = bank modulo 8); else every other pair, the columns modulo 16
                const int bank = lane & (C::kWarpCells - 1);
                int cy = k, cx = (bank + 4 * k) & 7;
                if constexpr (C::kSplit == 2) {
                    // cx = bank + 4 cy modulo 16 is a column for two of four rows in turn: from -bank / 4 on
                    cy = ((k & 1) - (bank >> 2) + ((bank >> 2) == 0 ? 0 : 4)) & 3;
                    cx = (bank + 4 * cy) & 15;
                    cy += (k & 2) * 2;
                }
                const int cell = cy * 8 + cx;
                keys[k] = sh.count[cz * 64 + cell] << 6 | cell;
            }
#pragma unroll
            for (int i = 1; i < C::kRounds; ++i)
#pragma unroll
                for (int j = i; j > 0; --j) {
                    const int a = keys[j - 1], b = keys[j];
                    keys[j - 1] = max(a, b);
                    keys[j] = min(a, b);
                }
            __syncwarp();
            if (part == 0)
#pragma unroll
                for (int k = 0; k < C::kRounds; ++k) {
                    sh.order[cz][k * C::kWarpCells + lane] = (unsigned char)(keys[k] & 63);
                    sh.count[cz * 64 + (keys[k] & 63)] = 0;
                }
            __syncwarp();
        }
#pragma unroll 1
        for (int round = 0; round < C::kRounds; ++round) {
            const int here = sh.order[cz][round * C::kWarpCells + (lane & (C::kWarpCells - 1))], cx = here & 7, cy = here >> 3, cell = cz * 64 + here;
            int p = sh.head[cell];
            if (!__any_sync(0xffffffffu, p != kChainEnd)) break;
            if (part == 0) sh.head[cell] = kChainEnd;
            u64 acc[C::kPlanes][4][4];
            float wacc[C::kPlanes][4][4];
#pragma unroll
            for (int k = 0; k < C::kPlanes; ++k)
#pragma unroll
                for (int y = 0; y < 4; ++y)
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        acc[k][y][x] = 0ull;
                        wacc[k][y][x] = 0.f;
                    }
            while (p != kChainEnd) {
                const float4 a = sh.a[p];
                const float2 u = sh.v[p];
                const float w = WEIGHTS ? sh.w[p] : 0.f;
                p = __float_as_int(a.w);
                float wx[4], wy[4], wz[C::kPlanes];
                cubic_weights(a.x, wx);
                cubic_weights(a.y, wy);
                if constexpr (C::kSplit == 2) {
                    // planes in the order outer, inner: of the upper half those of 1 - f
                    const float f = part ? 1.f - a.z : a.z;
                    wz[0] = cubic_weight_k<0>(f);
                    wz[1] = cubic_weight_k<1>(f);
                } else {
                    const float f = part >= 2 ? 1.f - a.z : a.z;
                    wz[0] = part == 0 || part == 3 ? cubic_weight_k<0>(f) : cubic_weight_k<1>(f);
                }
                const u64 u2 = pack2(u.x, u.y);
#pragma unroll
                for (int k = 0; k < C::kPlanes; ++k)
#pragma unroll
                    for (int y = 0; y < 4; ++y) {
                        const float f = wz[k] * wy[y];
                        const u64 q2 = fmul2(u2, pack2(f, f));
                        const float fw = w * fabsf(f);
#pragma unroll
                        for (int x = 0; x < 4; ++x) {
                            acc[k][y][x] = fma2(q2, pack2(wx[x], wx[x]), acc[k][y][x]);
                            if (WEIGHTS) wacc[k][y][x] = fmaf(fw, fabsf(wx[x]), wacc[k][y][x]);
                        }
                    }
            }
            // footprint plane of acc[k]
            auto plane = [&](int k) { return C::kSplit == 2 ? (part ? 3 - k : k) : part; };
            __syncwarp();
#pragma unroll
            for (int y = 0; y < 4; ++y)
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    float2 old[C::kPlanes];
                    float old_w[C::kPlanes];
                    int at[C::kPlanes];
#pragma unroll
                    for (int k = 0; k < C::kPlanes; ++k) {
                        at[k] = plane(k) * C::kPlane + (cy + y) * C::kRow + cx + x;
                        old[k] = sum[at[k]];
                        old_w[k] = WEIGHTS ? wsum[at[k]] : 0.f;
                    }
#pragma unroll
                    for (int k = 0; k < C::kPlanes; ++k) {
                        float re, im;
                        unpack2(acc[k][y][x], re, im);
                        sum[at[k]] = make_float2(old[k].x + re, old[k].y + im);
                        if (WEIGHTS) wsum[at[k]] = old_w[k] + wacc[k][y][x];
                    }
                    __syncwarp();
                }
        }
        __syncthreads();
        if (sh.queue.batch[s & 3].w) {
            // the layers' sums to the volume; cleared for the next item (whose first sums follow the next batch's barrier)
            const CellBrick brick = cell_brick<D>(pl, sh.queue.batch[s & 3].x);
            for (int t = tid; t < C::kSX * C::kSY * C::kSZ; t += C::kThreads) {
                const int row = t / C::kSX, x = t - row * C::kSX, z = row / C::kSY, y = row - z * C::kSY;
                float2 u = make_float2(0.f, 0.f);
                float f = 0.f;
                for (int l = max(0, z - 3); l <= min(z, D::kZ - 1); ++l) {
                    const int at = (z - l) * C::kPlane + y * C::kRow + x;
                    const float2 m = sh.sum[l][at];
                    sh.sum[l][at] = make_float2(0.f, 0.f);
                    u.x += m.x;
                    u.y += m.y;
                    if (WEIGHTS) {
                        f += sh.wsum[l][at];
                        sh.wsum[l][at] = 0.f;
                    }
                }
                if (u.x == 0.f && u.y == 0.f && f == 0.f) continue;
                scatter_voxel<3, DUP>(g, to, (long long)brick.b * g.vol_elems, brick.x - 1 + x, brick.y - 1 + y, brick.z - 1 + z, u.x, u.y, f);
            }
        }
    }
    if (odd) ws.header[5] = 1;
}

// ---- calls whose lists are left aside ---------------------------------------------------------------------------
// Poses may put a brick's pixels into a few of its cells; then most of the threads above have nothing to add, and the kernels without
// lists are faster (their reductions fall on few sectors).  The poses are on the device, so list_setup_kernel finds out, the kernels above
// return at once and the ones here run instead (Gate).  Plain kernels take several tiles to a block, as a grid whose blocks return at
// once takes 0.5-1 ns a block (0.2 ms for the 400,000 tiles of 10,000 slices of 128 x 65); persistent blocks that draw tickets are 5-18 % slower
// where they run.  10,000 slices of 128 x 65, weighted, linear: ten poses from lists
// 3.77 ms, without 2.19; tilt series in steps of 3 degrees 1.98 and 1.46; of one pose 3.71 and 2.60.
// x = `tiles` tiles of a slice, (y, z) = the slice.
template <int DIM, bool CUBIC, bool DUP>
__global__ void __launch_bounds__(kBlockThreads)
gated_scatter_kernel(const float2* __restrict__ proj, const float* __restrict__ rot, const float* __restrict__ shifts, float2* __restrict__ vol,
                     const SliceGeom g, int tiles, const Gate gate) {
    if (gate.shut()) return;
    for (int x = (int)blockIdx.x * tiles, end = min(x + tiles, g.tiles_i * g.tiles_j); x < end; ++x)
        backproject_forw<DIM, CUBIC, false, DUP, float>(g, block_work(g, x, (int)blockIdx.y, (int)blockIdx.z), proj, nullptr, rot, shifts, vol, nullptr);
}
template <int DIM, bool CUBIC>
__global__ void __launch_bounds__(kBlockThreads)
gated_interleaved_kernel(const float2* __restrict__ proj, const float* __restrict__ weights, const float* __restrict__ rot, const float* __restrict__ shifts,
                         float4* __restrict__ accum, const SliceGeom g, int tiles, const Gate gate) {
    if (gate.shut()) return;
    for (int x = (int)blockIdx.x * tiles, end = min(x + tiles, g.tiles_i * g.tiles_j); x < end; ++x)
        backproject_forw_interleaved<DIM, CUBIC>(g, block_work(g, x, (int)blockIdx.y, (int)blockIdx.z), proj, weights, rot, shifts, accum);
}
__global__ void __launch_bounds__(256)
gated_zero_kernel(float4* __restrict__ to, size_t n, const Gate gate) {
    if (gate.shut()) return;
    for (size_t t = (size_t)blockIdx.x * 256 + threadIdx.x; t < n; t += (size_t)gridDim.x * 256) to[t] = make_float4(0.f, 0.f, 0.f, 0.f);
}

}  // namespace b200proj
