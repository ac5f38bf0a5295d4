// Brick-stationary scatters (fp32, cubic taps): gradient of the projection with respect to the volume, and
// back-projection.  The plain kernels send every tap to L2 as a reduction and sit on the rate at which reductions
// leave the SMs.  Here a brick's sums are kept in shared memory and leave once per work item.
//
// Shared-memory float atomics are compare-and-swap loops (6.5 clocks per warp and float); plain load, add, store is
// 4.3 clocks per warp and complex number, but then only one warp may touch a sum.  So a brick is cut along z into
// slabs, each with its own sums (halo planes included) and its own ADDING warp; the other warps of the block WALK over
// the slices (brick_walk) and put each pixel into the ring of its slab.  A ring is a few chunks of 32 pixels, each with
// an mbarrier that completes when its 32 pixels are written, and a count of the chunks that the adding warp has taken
// (a count and not a second mbarrier: the walkers' reservations can be more than one phase ahead), so that no warp
// waits for any other but through a full or empty ring.
//
// An adding warp takes a chunk, one pixel per lane, and every lane its taps in an order that starts at the lane's own
// class (x & 3, y & 3, z & 3) -- a cubic footprint holds every class once --, two taps a step: the 32 lanes hold 64
// different classes then, hence 64 different voxels, whatever pixels they hold.  So no two lanes add to the same voxel
// between two synchronisations of the warp, and the 8-byte sums meet no bank conflicts (of the 4-byte sums of the weights
// those of lanes 16 apart can meet in a bank).  2D reconstructions are cut into tiles; a
// tile's pixels go to the adding warps in turn, each of which has its own sums (two copies: a 4 x 4 footprint has 16
// classes, so the halves of the warp are kept apart).
//
// Measured on B200: the scatter of 4,096 slices of 256 x 129 into a box-512 gradient 14.4 ms (plain kernel) -> 5.97 ms,
// 2,501 weighted slices of box 90 into box 180 1.61 -> 0.75 ms.  What bounds it, from timers around the waits, in
// shares of the kernel's time: without weights the walk (the walking warps walk for 67 % and wait for room for 7 %, the
// adding warps add for 53 % and wait for chunks for 37 %), with weights the adding (64 % and 24 %, walking warps 43 % and
// 27 %); flushes are 6-7 %.  A step of 64 taps is a chain of load, add, store: 58 clocks alone, 100 beside the other warps
// of the SM (126 with weights), which use 56 % of the issue slots.  An SM holds 12 slabs of 13 x 13 x 4 sample
// positions (16 x 16 x 7 sums), 8 with weights.  Measured slower for that scatter: 10 slabs of 5
// planes 6.1 ms, 8 slabs of 8 planes 6.4 ms, one block of 14 walkers and 10 slabs 6.6 ms, one adding warp per block
// with a barrier for each hand-over 7.8 ms, and pixels of a full ring sent to L2 as reductions by the walkers 7.6 ms
// (that starves the adding warps).  For linear taps (2 x 2 x 2 classes, overlapping pixels one after the other) the
// same scheme took 44-46 ps per pixel where the plain kernels take 33.
//
// Calls with more pixels per brick, linear ones included, run from pixel lists (cell_scatter.cuh), which take 42 instead of 56 ps per
// pixel of the scatter above; these kernels have the calls whose bricks hold too few pixels for a cell's sums to pay
// (list_scatter_plan in b200proj.cu), and those whose workspace has no room for a list.
#pragma once

#include "brick_kernels.cuh"

namespace b200proj {

// ---- shared memory and mbarriers -----------------------------------------------------------------------------
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned long long lds64(unsigned a) {
    unsigned long long v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts64(unsigned a, unsigned long long v) { asm volatile("st.shared.b64 [%0], %1;" ::"r"(a), "l"(v) : "memory"); }
__device__ __forceinline__ float lds32(unsigned a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts32(unsigned a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar, unsigned count) {
    asm volatile("{ .reg .b64 state; mbarrier.arrive.shared::cta.b64 state, [%0], %1; }" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
// Every wait ends by construction (see brick_scatter_kernel).  Should one not, it gives up: the block then writes NaN
// into the bricks that it could not finish, so that the loss shows in the result, and the kernel returns.  The limit is
// time spent polling; a gap between two polls counts 1 ms at most (a block that was not running loses no patience).
struct Patience {
    unsigned long long last = 0ull, spent = 0ull, limit;
    __device__ explicit Patience(int ms) : limit((unsigned long long)ms * 1000000ull) {}
    __device__ __forceinline__ bool over() {
        unsigned long long now;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
        if (last != 0ull) spent += min(now - last, 1000000ull);
        last = now;
        return spent >= limit;
    }
};
// Wait for the phase of the given parity; false: given up, by this wait or another of the block.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, int* gave_up, int limit_ms) {
    Patience patience(limit_ms);
    while (true) {
        unsigned ready;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(ready) : "r"(smem_addr(bar)), "r"(parity) : "memory");
        if (ready) return true;
        if (*(volatile int*)gave_up) return false;
        if (patience.over()) {
            *(volatile int*)gave_up = 1;
            return false;
        }
    }
}
// Wait until *count exceeds `below`, likewise.
__device__ __forceinline__ bool count_wait(const int* count, int below, int* gave_up, int limit_ms) {
    Patience patience(limit_ms);
    while (*(const volatile int*)count <= below) {
        if (*(volatile int*)gave_up) return false;
        if (patience.over()) {
            *(volatile int*)gave_up = 1;
            return false;
        }
        __nanosleep(32);
    }
    return true;
}

// ---- sizes --------------------------------------------------------------------------------------------------
// kX x kY sample positions, kSlabs slabs of kSlab planes of them; kBlocks blocks per SM of kWalkers + kSlabs warps.
template <int DIM, bool WEIGHTS>
struct ScatterSizes;
template <> struct ScatterSizes<3, false> { static constexpr int kX = 13, kY = 13, kSlab = 4, kSlabs = 6, kWalkers = 6, kBlocks = 2, kRing = 4; };
template <> struct ScatterSizes<3, true> { static constexpr int kX = 13, kY = 13, kSlab = 4, kSlabs = 4, kWalkers = 6, kBlocks = 2, kRing = 4; };

// 2D: kSlabs counts adding warps, each with two copies of the tile's sums (kSlab = 0).  A pixel has 16 taps there, so the
// walk weighs more: 27 M pixels of box 128, gradient, 5 + 7 warps 0.73 ms, 4 + 8 0.79, 6 + 6 0.87; weighted 4 + 8 0.97, 5 + 7 on
// smaller tiles 0.92 (but 1.27 against 0.98 for box 32), 6 + 6 1.02.
template <> struct ScatterSizes<2, false> { static constexpr int kX = 29, kY = 29, kSlab = 0, kSlabs = 5, kWalkers = 7, kBlocks = 2, kRing = 4; };
template <> struct ScatterSizes<2, true> { static constexpr int kX = 25, kY = 25, kSlab = 0, kSlabs = 4, kWalkers = 8, kBlocks = 2, kRing = 4; };

template <int DIM, bool WEIGHTS>
struct Scatter : ScatterSizes<DIM, WEIGHTS> {
    using Z = ScatterSizes<DIM, WEIGHTS>;
    using Brick = BrickDims<Z::kX, Z::kY, Z::kSlab * Z::kSlabs>;
    static constexpr int kThreads = (Z::kWalkers + Z::kSlabs) * 32;
    static constexpr int kTX = Z::kX + 3, kTY = Z::kY + 3, kTZ = DIM == 3 ? Z::kSlab + 3 : 2;   // of one slab, halo included
    static_assert(kTX % 4 == 0 && kTY % 4 == 0 && (DIM == 2 || Z::kSlab >= 3) && Z::kRing >= 2, "whole cells; two slabs share a plane at most");
    static constexpr int kPlane = kTX * kTY, kVoxels = kPlane * kTZ;
    struct Slab {
        float2 sum[kVoxels];
        float wsum[WEIGHTS ? kVoxels : 4];
    };
    struct Ring {
        float4 a[Z::kRing * 32];                    // fx, fy, fz, x | y << 8 | z << 16 | flags << 24
        float2 v[Z::kRing * 32];
        float w[WEIGHTS ? Z::kRing * 32 : 4];
        unsigned long long full[Z::kRing];
        int tail, taken;                            // places reserved, chunks taken so far
        int pad[2];
    };
    struct Shared {
        Slab slab[Z::kSlabs];
        Ring ring[Z::kSlabs];
        BrickBlock<1, 64> walk[Z::kWalkers];
        int item, done, gave_up;
    };
    // place of the voxel (x, y, z) of a slab (2D: copy z): 4 x 4 cells of a plane are contiguous
    __device__ static __forceinline__ int place(int x, int y, int z) { return z * kPlane + 4 * (y & 3) + kTX * 4 * (y >> 2) + x + 12 * (x >> 2); }
};
constexpr unsigned kItemEnds = 1u << 24;        // flag of a ring's last entry of an item

// ---- adding 32 pixels, one per lane ---------------------------------------------------------------------------
// A lane without a pixel adds zeros (its classes are its own).
template <bool WEIGHTS>
__device__ __forceinline__ void brick_add_2d(typename Scatter<2, WEIGHTS>::Slab& sb, const float4 a, float2 v, float wv) {
    using C = Scatter<2, WEIGHTS>;
    using u64 = unsigned long long;
    const int lane = threadIdx.x & 31;
    const unsigned at = __float_as_uint(a.w);
    const int lx = at & 255, ly = at >> 8 & 255, rx = lx & 3, ry = ly & 3;
    // lanes 16 apart hold the same class: each half of the warp has its own copy
    const unsigned base = (unsigned)((lane >> 4) * C::kPlane + (ly >> 2) * (C::kTX * 4) + (lx >> 2) * 16) * 8u + smem_addr(sb.sum);
    unsigned ox[4];
    float wx[4], wy[4];
    cubic_weights(a.x, wx);
    rotate4(wx, (lane - lx) & 3);
    cubic_weights(a.y, wy);
    rotate4(wy, ((lane >> 2) - ly) & 3);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int ax = (lane + s) & 3;
        ox[s] = (unsigned)(ax * 8 + (ax < rx ? 128 : 0)) + base;
    }
    const u64 v2 = pack2(v.x, v.y);
    const unsigned half = (smem_addr(sb.sum) >> 1) - smem_addr(sb.wsum);      // weights: half the distance
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const int ay = ((lane >> 2) + b) & 3;
        const unsigned oy = (unsigned)(ay * 32 + (ay < ry ? C::kTX * 32 : 0));
        const u64 q = fmul2(pack2(wy[b], wy[b]), v2);
        const float f = WEIGHTS ? wv * fabsf(wy[b]) : 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned s0 = oy + ox[k];
            const u64 u = lds64(s0);
            if (WEIGHTS) {
                const unsigned t0 = (s0 >> 1) - half;
                const float g0 = lds32(t0);
                sts64(s0, fma2(pack2(wx[k], wx[k]), q, u));
                sts32(t0, fmaf(fabsf(wx[k]), f, g0));
            } else {
                sts64(s0, fma2(pack2(wx[k], wx[k]), q, u));
            }
            __syncwarp();
        }
    }
}

template <bool WEIGHTS>
__device__ __forceinline__ void brick_add(typename Scatter<3, WEIGHTS>::Slab& sb, const float4 a, float2 v, float wv) {
    using C = Scatter<3, WEIGHTS>;
    using u64 = unsigned long long;
    constexpr int kPlane = C::kPlane;
    const int lane = threadIdx.x & 31;
    const unsigned at = __float_as_uint(a.w);
    const int lx = at & 255, ly = at >> 8 & 255, lz = at >> 16 & 255;
    const int rx = lx & 3, ry = ly & 3, tx = (lane - lx) & 3, ty = ((lane >> 2) - ly) & 3, tz = (2 * (lane >> 4) - lz) & 3;
    unsigned ox[4], oy[4], oz[4];
    const unsigned base = (unsigned)(lz * kPlane + (ly >> 2) * (C::kTX * 4) + (lx >> 2) * 16) * 8u + smem_addr(sb.sum);
    float wx[4], wy[4], wz[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int ax = (lane + s) & 3, ay = ((lane >> 2) + s) & 3;
        ox[s] = (unsigned)(ax * 8 + (ax < rx ? 128 : 0));
        oy[s] = (unsigned)(ay * 32 + (ay < ry ? C::kTX * 32 : 0));
        oz[s] = (unsigned)(((tz + s) & 3) * kPlane * 8) + base;
    }
    cubic_weights(a.x, wx);
    rotate4(wx, tx);
    cubic_weights(a.y, wy);
    rotate4(wy, ty);
    cubic_weights(a.z, wz);
    rotate4(wz, tz);
    const u64 v2 = pack2(v.x, v.y);
    u64 wx2[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) wx2[s] = pack2(wx[s], wx[s]);
    const unsigned half = (smem_addr(sb.sum) >> 1) - smem_addr(sb.wsum);      // weights: half the distance
#pragma unroll
    for (int c = 0; c < 4; c += 2) {
        const u64 p0 = fmul2(pack2(wz[c], wz[c]), v2), p1 = fmul2(pack2(wz[c + 1], wz[c + 1]), v2);
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const u64 wy2 = pack2(wy[b], wy[b]);
            const u64 q0 = fmul2(wy2, p0), q1 = fmul2(wy2, p1);
            const unsigned a0 = oz[c] + oy[b], a1 = oz[c + 1] + oy[b];
            float f0 = 0.f, f1 = 0.f;
            if (WEIGHTS) {
                f0 = wv * fabsf(wz[c] * wy[b]);
                f1 = wv * fabsf(wz[c + 1] * wy[b]);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const unsigned s0 = a0 + ox[k], s1 = a1 + ox[k];
                const u64 u0 = lds64(s0), u1 = lds64(s1);
                if (WEIGHTS) {
                    const unsigned t0 = (s0 >> 1) - half, t1 = (s1 >> 1) - half;
                    const float g0 = lds32(t0), g1 = lds32(t1);
                    sts64(s0, fma2(wx2[k], q0, u0));
                    sts64(s1, fma2(wx2[k], q1, u1));
                    sts32(t0, fmaf(fabsf(wx[k]), f0, g0));
                    sts32(t1, fmaf(fabsf(wx[k]), f1, g1));
                } else {
                    sts64(s0, fma2(wx2[k], q0, u0));
                    sts64(s1, fma2(wx2[k], q1, u1));
                }
                __syncwarp();
            }
        }
    }
}

// Sums of a finished item to the volume, by the scatter's rules (Friedel mirror with conjugation, taps outside the
// stored half-volume dropped, DUP: the conjugate also to the Friedel partner of a voxel on the c == 0 plane); cleared
// for the next item.  INTERLEAVED: into 16-byte (re, im, weight, 0) voxels.  LOST: sums of the item are missing; NaN.
template <int DIM, bool WEIGHTS, bool DUP, bool INTERLEAVED>
__device__ __forceinline__ void brick_flush(const SliceGeom& g, typename Scatter<DIM, WEIGHTS>::Shared& sh, float2* __restrict__ vol, float* __restrict__ wvol,
                                            float4* __restrict__ accum, int X0, int Y0, int Z0, bool lost) {
    using C = Scatter<DIM, WEIGHTS>;
    auto add = [&](int off, float re, float im, float w) {
        if (INTERLEAVED) {
            red_add_v4(accum + off, re, im, w, 0.f);
        } else {
            red_add_v2(vol + off, re, im);
            if (WEIGHTS) red_add(wvol + off, w);
        }
    };
    // 3D: planes that two slabs share are added up first (the first three planes of a slab are the last of the one
    // below); 2D: the copies of all adding warps
    for (int t = (int)threadIdx.x; t < (DIM == 3 ? C::kSlab * C::kSlabs + 3 : 1) * C::kPlane; t += C::kThreads) {
        const int x = t % C::kTX, row = t / C::kTX, y = row % C::kTY, z = row / C::kTY;
        float2 v = make_float2(0.f, 0.f);
        float w = 0.f;
        auto take = [&](typename C::Slab& sb, int at) {
            const float2 u = sb.sum[at];
            sb.sum[at] = make_float2(0.f, 0.f);
            v.x += u.x;
            v.y += u.y;
            if (WEIGHTS) {
                w += sb.wsum[at];
                sb.wsum[at] = 0.f;
            }
        };
        if constexpr (DIM == 3) {
            const int last = min(z / C::kSlab, C::kSlabs - 1), first = max(0, z - 3) / C::kSlab;
            for (int s = first; s <= last; ++s) take(sh.slab[s], C::place(x, y, z - s * C::kSlab));
        } else {
#pragma unroll
            for (int s = 0; s < C::kSlabs; ++s) {
                take(sh.slab[s], C::place(x, y, 0));
                take(sh.slab[s], C::place(x, y, 1));
            }
        }
        if (lost) v.x = v.y = w = __int_as_float(0x7fffffff);
        if (v.x == 0.f && v.y == 0.f && w == 0.f) continue;
        bool m;
        const int c = scatter_col(g, X0 - 1 + x, m), r = scatter_line(g, Y0 - 1 + y, m), d = DIM == 3 ? scatter_line(g, Z0 - 1 + z, m) : 0;
        if (c < 0 || r < 0 || d < 0) continue;
        if (m) v.y = -v.y;
        add((d * g.R + r) * g.Rh + c, v.x, v.y, w);
        if (DUP && c == 0) {
            const int r2 = r == 0 ? 0 : g.R - r, d2 = d == 0 ? 0 : g.R - d;
            if (r2 != r || d2 != d) add((d2 * g.R + r2) * g.Rh, v.x, -v.y, w);
        }
    }
}

// No wait can last: a walking warp writes each ring as soon as that ring has room, so the lowest place of a ring that is
// not written yet waits only for chunks before its own (a ring has more than one), all of which are written and will be
// taken; the last warp to finish its walk fills every ring up to a whole chunk.
template <int DIM, bool WEIGHTS, bool DUP, bool INTERLEAVED>
__global__ void __launch_bounds__(Scatter<DIM, WEIGHTS>::kThreads, Scatter<DIM, WEIGHTS>::kBlocks)
brick_scatter_kernel(const float2* __restrict__ proj, const float* __restrict__ weights, const float* __restrict__ rot,
                     const float* __restrict__ shifts, float2* __restrict__ vol, float* __restrict__ wvol, float4* __restrict__ accum,
                     BrickWork ws, const SliceGeom g, const BrickPlan pl, Gate gate) {
    if (gate.shut()) return;
    using C = Scatter<DIM, WEIGHTS>;
    extern __shared__ __align__(16) unsigned char dyn[];
    typename C::Shared& sh = *reinterpret_cast<typename C::Shared*>(dyn);
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int t = (int)threadIdx.x; t < (int)(sizeof(sh.slab) / 16); t += C::kThreads) reinterpret_cast<float4*>(sh.slab)[t] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (threadIdx.x < C::kSlabs) {
        typename C::Ring& q = sh.ring[threadIdx.x];
        for (int c = 0; c < C::kRing; ++c) mbar_init(&q.full[c], 32);
        q.tail = q.taken = 0;
    }
    if (threadIdx.x == 0) sh.gave_up = 0;
    int slot = 0, taken = 0;                                // adding warps: next chunk of the ring, its parity, chunks taken
    unsigned parity = 0;
    const int items = brick_items(ws);
    bool lost = false;                                      // a wait of this block gave up: its rings are of no use any more
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) {
            sh.item = atomicAdd(ws.header + 2, 1);
            sh.done = 0;
        }
        __syncthreads();
        const int item = sh.item;
        if (item >= items) break;
        // the item's share of the slices that are not for the bricks: plain scatter
        for (int k = (int)((long long)g.BP * item / items), k_end = (int)((long long)g.BP * (item + 1) / items); k < k_end; ++k) {
            const int b = k / g.P, p = k - b * g.P;
            if (brick_has_slice(ws, k)) continue;
            const int nj = (g.Nh + 7) / 8, ni = (g.N + 3) / 4;
            for (int patch = warp; patch < ni * nj; patch += C::kThreads / 32) {
                BlockWork w;
                w.b = b;
                w.p = p;
                w.i = patch / nj * 4 + (lane >> 3);
                w.j = patch % nj * 8 + (lane & 7);
                w.in_image = w.i < g.N && w.j < g.Nh;
                w.pix = (size_t)k * (size_t)g.slice_pixels + (size_t)(w.i * g.Nh + w.j);
                Pixel px;
                float2 v;
                float wv;
                const bool active = backproject_pixel<DIM, WEIGHTS>(g, w, proj, weights, rot, shifts, px, v, wv);
                const size_t at = (size_t)b * g.vol_elems;
                scatter_coop<DIM, true, WEIGHTS, DUP, INTERLEAVED>(g, INTERLEAVED ? nullptr : vol + at, WEIGHTS && !INTERLEAVED ? wvol + at : nullptr,
                                                                  INTERLEAVED ? accum + at : nullptr, px, active, v, wv);
            }
        }
        const int4 it = brick_item(ws, pl, item);
        const int X0 = pl.lo[0] + (it.x & 1023) * C::Brick::x, Y0 = pl.lo[1] + ((it.x >> 10) & 1023) * C::Brick::y, Z0 = pl.lo[2] + (it.x >> 20) * C::Brick::z;
        if (!lost && warp < C::kWalkers) {
            const BrickWarp& sw = sh.walk[warp].warp[0];
            // places [first, first + n) of a ring are written: its chunks count them
            auto arrive = [&](typename C::Ring& q, int first, int n) {
                const int c0 = first >> 5, n0 = min(n, 32 - (first & 31));
                mbar_arrive(&q.full[c0 % C::kRing], (unsigned)n0);
                if (n > n0) mbar_arrive(&q.full[(c0 + 1) % C::kRing], (unsigned)(n - n0));
            };
            auto write = [&](typename C::Ring& q, int place, const float4& a, float2 v, float w) {
                const int at = place % (C::kRing * 32);
                q.a[at] = a;
                q.v[at] = v;
                if (WEIGHTS) q.w[at] = w;
            };
            // the previous window's pixels, whose values are still on their way from memory
            int h_slab = -1, turn = warp % C::kSlabs;
            float4 h_a = make_float4(0.f, 0.f, 0.f, 0.f);
            float2 h_v = make_float2(0.f, 0.f), h_ph = make_float2(1.f, 0.f);
            float h_w = 0.f;
            // Lane s reserves places in ring s; when all of them are free, all lanes write at once.  Else ring by ring as
            // they become free, never waiting for one while another could be written.
            auto put = [&] {
                const bool mine = h_slab >= 0;
                if (mine && g.has_shift) h_v = cmul_conj(h_v, h_ph);
                int n = 0, rank = 0, first = 0;
#pragma unroll
                for (int s = 0; s < C::kSlabs; ++s) {
                    const unsigned m = __ballot_sync(kFull, h_slab == s);
                    if (lane == s) n = __popc(m);
                    if (h_slab == s) rank = __popc(m & ((1u << lane) - 1u));
                }
                if (n > 0) first = atomicAdd(&sh.ring[lane].tail, n);
                const int place = __shfl_sync(kFull, first, max(h_slab, 0)) + rank;
                typename C::Ring& q = sh.ring[max(h_slab, 0)];
                const bool room = n == 0 || *(volatile int*)&sh.ring[lane].taken > ((first + n - 1) >> 5) - C::kRing;
                if (__all_sync(kFull, room)) {
                    if (mine) write(q, place, h_a, h_v, h_w);
                    __syncwarp();
                    if (n > 0) arrive(sh.ring[lane], first, n);
                    return;
                }
                Patience patience(pl.wait_ms);
                for (unsigned left = __ballot_sync(kFull, n > 0); left != 0u;) {
                    const bool now = (left >> lane & 1u) != 0u && *(volatile int*)&sh.ring[lane].taken > ((first + n - 1) >> 5) - C::kRing;
                    const unsigned ready = __ballot_sync(kFull, now);
                    if (mine && (ready >> h_slab & 1u) != 0u) write(q, place, h_a, h_v, h_w);
                    __syncwarp();
                    if (now) arrive(sh.ring[lane], first, n);
                    left &= ~ready;
                    if (ready == 0u) {
                        if (patience.over()) *(volatile int*)&sh.gave_up = 1;
                        if (__any_sync(kFull, *(volatile int*)&sh.gave_up != 0)) return;
                        __nanosleep(64);
                    }
                }
            };
            brick_walk<typename C::Brick>(g, ws.recs, ws.shifts, sh.walk[warp], X0, Y0, Z0, it.z, it.w, warp, C::kWalkers,
                                          [&](bool active, int slot_, int i, int j, const Pixel& px, int lx, int ly, int lz) {
                active = active && !(j == 0 && i >= g.N / 2);
                float2 v = make_float2(0.f, 0.f);
                float w = 0.f;
                if (active) {
                    const size_t pix = (size_t)sw.slice[slot_] * (size_t)g.slice_pixels + (size_t)(i * g.Nh + j);
                    v = __ldg(proj + pix);
                    if (WEIGHTS) w = __ldg(weights + pix);
                }
                put();
                int s = 0;
                if constexpr (DIM == 3) s = lz / C::kSlab;
                else s = turn = turn + 1 < C::kSlabs ? turn + 1 : 0;                // windows are dealt to the adding warps in turn
                h_slab = active ? s : -1;
                h_a = make_float4(px.c - floorf(px.c), px.r - floorf(px.r), DIM == 3 ? px.d - floorf(px.d) : 0.f,
                                  __uint_as_float((unsigned)(lx | ly << 8 | (DIM == 3 ? lz - s * C::kSlab : 0) << 16)));
                h_v = v;
                h_w = w;
                if (g.has_shift) {
                    const float4 rc = sw.slots[slot_][1];
                    h_ph = phase_ramp(g, px, rc.z, rc.w);
                }
            });
            put();
            __syncwarp();
            int finished = 0;
            if (lane == 0) {
                __threadfence_block();
                finished = atomicAdd(&sh.done, 1) + 1;
                __threadfence_block();
            }
            if (__shfl_sync(kFull, finished, 0) == C::kWalkers) {
                for (int s = 0; s < C::kSlabs; ++s) {
                    typename C::Ring& q = sh.ring[s];
                    const int first = *(volatile int*)&q.tail, n = 32 - (first & 31);
                    __syncwarp();
                    if (lane == 0) *(volatile int*)&q.tail = first + n;
                    if (!__all_sync(kFull, count_wait(&q.taken, (first >> 5) - C::kRing, &sh.gave_up, pl.wait_ms))) break;
                    if (lane < n) write(q, first + lane, make_float4(0.f, 0.f, 0.f, __uint_as_float(lane == n - 1 ? kItemEnds : 0u)), make_float2(0.f, 0.f), 0.f);
                    __syncwarp();
                    if (lane == 0) arrive(q, first, n);
                }
            }
        } else if (!lost) {
            typename C::Ring& q = sh.ring[warp - C::kWalkers];
            typename C::Slab& sb = sh.slab[warp - C::kWalkers];
            bool ends = false;
            while (!ends) {
                if (!__all_sync(kFull, mbar_wait(&q.full[slot], parity, &sh.gave_up, pl.wait_ms))) break;
                const float4 a = q.a[slot * 32 + lane];
                const float2 v = q.v[slot * 32 + lane];
                const float w = WEIGHTS ? q.w[slot * 32 + lane] : 0.f;
                __syncwarp();
                if (lane == 0) {
                    __threadfence_block();
                    *(volatile int*)&q.taken = ++taken;
                }
                if (++slot == C::kRing) { slot = 0; parity ^= 1u; }
                ends = (__shfl_sync(kFull, __float_as_uint(a.w), 31) & kItemEnds) != 0u;
                if constexpr (DIM == 3) brick_add<WEIGHTS>(sb, a, v, w);
                else brick_add_2d<WEIGHTS>(sb, a, v, w);
            }
        }
        __syncthreads();
        lost = sh.gave_up != 0;
        const size_t at = (size_t)it.y * g.vol_elems;
        brick_flush<DIM, WEIGHTS, DUP, INTERLEAVED>(g, sh, INTERLEAVED ? nullptr : vol + at, WEIGHTS && !INTERLEAVED ? wvol + at : nullptr,
                                                      INTERLEAVED ? accum + at : nullptr, X0, Y0, Z0, lost);
    }
    if (threadIdx.x == 0 && lost) ws.header[3] = 1;
}

}  // namespace b200proj
