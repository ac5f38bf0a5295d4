// Pixel lists (fp32): the pixels of a call's slices, sorted by the brick of the volume that their sample position lies in.
// The kernels that add a brick up on chip (cell_scatter.cuh) then read the brick's pixels off a list and test nothing.
// A list entry is 4 bytes, slice and (row, column) as bit fields; whoever reads it works out the sample position again,
// with the same operations and hence the same bits.
//
// The volume holds half of a Hermitian spectrum, so a sample at x with x_c < 0 is the conjugate of the one at -x.  Samples
// whose whole footprint has c < 0 are folded over: their pixels join those of -x, which halves the bricks and doubles
// the pixels in each.  Footprints that touch c = 0 stay where they are (the edge rules tell the two sides apart there),
// for which the grid starts a brick below.
//
// A call runs as
//   list_setup_kernel    the pixels inside the cutoff, in patches of 16 x 4; a 32-byte record per slice; whether the poses crowd
//   list_pixels_kernel   counts the pixels of each brick (COUNT), later writes their entries
//   list_plan_kernel     a place in the list for each brick, work items of at most `most` pixels of one brick
#pragma once

#include "fourier_slice_kernels.cuh"

namespace b200proj {

// Cells (unit cubes of sample positions) of a brick: 8 x 8 x 8; 2D: of a tile, 16 x 16.  (Linear taps, bricks of 8 x 8 x 4: more bricks a
// slice meets, 25 % more time in both passes over the pixels.)
template <int DIM>
struct ListBrick;
template <> struct ListBrick<3> { static constexpr int kLogX = 3, kLogY = 3, kLogZ = 3, kFirst = -8; };
template <> struct ListBrick<2> { static constexpr int kLogX = 4, kLogY = 4, kLogZ = 0, kFirst = -16; };
// kFirst: first cell along c; samples with c < kFirst are folded over.

struct ListPlan {
    int n[3];               // bricks along x (column), y (row), z (plane)
    int lo[3];              // first cell of the grid along them
    int bits;               // of the largest of n
    float row_zero;         // 2^23 + N / 2 - 1: what a row of an entry is counted from
    float round[2];         // kRound less lo in bricks, of rows and planes
    float fit[3];           // samples below these stay in the grid
    float reach;            // frequency of the farthest listed pixel, times the oversampling
    int bricks, item_bricks;    // of all batch items, of one
    int bits_j, bits_i;     // of a list entry
    int first, slices;      // slices of this pass over the list: first .. first + slices
    int inside;             // pixels of a slice that are listed
    int pairs;              // room for their pairs
    int most;               // pixels of a work item
    int subs;               // counters of a brick (a power of two), for slices taken in turn
    unsigned spread, groups;    // of the counters, see list_counter; groups of 8 less one
    int probes;             // blocks of list_setup_kernel that look at how the pixels crowd
    float crowd;            // the lists are left aside when that finds fewer cells
    int run;                // slices of a block of list_pixels_kernel that counts in shared memory; 0: in global memory
    int turn;               // and of one that counts in global memory
    unsigned capacity;      // entries of the list
};

// Workspace: int header[64] {entries, work items, ticket, 0 (the brick scatters' status), slices that are not listed, 1: some pixel is
// not finite, slices with samples out of the grid, pairs, probed pixels of a brick, of a cell, -}, then what follows, each part on a 256-byte boundary.
struct ListWork {
    int* header;
    unsigned* count;        // pixels of each brick, at list_counter; after list_plan_kernel: where the next entry goes
    int4* items;            // {brick, first entry, entries, -}
    float4* poses;          // per slice of the call: {m00, m10, m20, m01}, {m11, m21, shift}; NaN: the slice is not listed
    unsigned* inside;       // pairs of neighbours in a row: what an entry says of the first pixel, (row frequency + N / 2 - 1) << bits_j
                            // | column (even), and which of the two are listed, 1 << 30 and 1 << 31
    unsigned* block_count;  // pixels of each brick in a block of list_pixels_kernel
    unsigned* list;
};

// Conversions between floats and integers run at an eighth of the rate of additions.  These are exact for |x| < 2^22.
constexpr float kRound = 12582912.f;        // 1.5 * 2^23: the unit in the last place is 1
constexpr int kRoundBits = 0x4b400000;
__device__ __forceinline__ float small_int_to_float(int k) { return __int_as_float(0x4b000000 | k) - 8388608.f; }       // 0 <= k < 2^23

struct ListSample {
    float kr, kc;
    float fc, fr, fd;       // sample position, folded: fractions
    int x, y, z;            // and the cell, from the grid's first
    bool folded;
};

// The sample position of a listed pixel, formed as pixel_setup does (lists are for factors of oversampling that are floats: with
// a conversion to double and back for the others in the kernels they took 10 % more time), and its cell.  What lies beyond 2^22 is out of the
// grid whatever it rounds to.
template <int DIM>
__device__ __forceinline__ ListSample list_sample(const SliceGeom& g, const ListPlan& pl, const float4& ra, const float4& rb, unsigned row, unsigned column) {
    ListSample s;
    s.kr = __int_as_float(0x4b000000 | (int)row) - pl.row_zero;
    s.kc = small_int_to_float((int)column);
    const float sc = mul_rn(s.kc, g.os_f), sr = mul_rn(s.kr, g.os_f);
    float c = add_rn(mul_rn(ra.x, sc), mul_rn(ra.w, sr));
    float r = add_rn(mul_rn(ra.y, sc), mul_rn(rb.x, sr));
    float d = DIM == 3 ? add_rn(mul_rn(ra.z, sc), mul_rn(rb.y, sr)) : 0.f;
    s.folded = c < (float)ListBrick<DIM>::kFirst;
    if (s.folded) {
        c = -c;
        r = -r;
        d = -d;
    }
    const float tc = __fadd_rd(c, kRound), tr = __fadd_rd(r, kRound), td = __fadd_rd(d, kRound);
    s.x = __float_as_int(tc) - (kRoundBits + pl.lo[0]);
    s.y = __float_as_int(tr) - (kRoundBits + pl.lo[1]);
    s.z = DIM == 3 ? __float_as_int(td) - (kRoundBits + pl.lo[2]) : 0;
    s.fc = c - (tc - kRound);
    s.fr = r - (tr - kRound);
    s.fd = DIM == 3 ? d - (td - kRound) : 0.f;
    return s;
}
// Bricks of a pair of pixels; -1: out of the grid, where no tap is inside the volume (fit: that no sample is).  A coordinate of the
// brick is one fused multiply-add rounded down, which loses nothing: the same as the cell's over the edge of a brick.
template <int DIM>
__device__ __forceinline__ void list_bricks(const SliceGeom& g, const ListPlan& pl, const float4& ra, const float4& rb, unsigned entry, int b, bool fit, int& first, int& second) {
    using L = ListBrick<DIM>;
    constexpr float kX = 1.f / (1 << L::kLogX), kY = 1.f / (1 << L::kLogY), kZ = 1.f / (1 << L::kLogZ);
    const float sr = mul_rn(__int_as_float(0x4b000000 | (int)(entry >> pl.bits_j)) - pl.row_zero, g.os_f);
    const float kc = small_int_to_float((int)(entry & ((1u << pl.bits_j) - 1u)));
    const float rc = mul_rn(ra.w, sr), rr = mul_rn(rb.x, sr), rd = DIM == 3 ? mul_rn(rb.y, sr) : 0.f;
    auto brick = [&](float column) {
        const float sc = mul_rn(column, g.os_f);
        float c = add_rn(mul_rn(ra.x, sc), rc), r = add_rn(mul_rn(ra.y, sc), rr), d = DIM == 3 ? add_rn(mul_rn(ra.z, sc), rd) : 0.f;
        if (c < (float)L::kFirst) {
            c = -c;
            r = -r;
            d = -d;
        }
        const int x = __float_as_int(__fmaf_rd(c, kX, kRound + 1.f)) - kRoundBits;
        const int y = __float_as_int(__fmaf_rd(r, kY, pl.round[0])) - kRoundBits;
        const int z = DIM == 3 ? __float_as_int(__fmaf_rd(d, kZ, pl.round[1])) - kRoundBits : 0;
        if (!fit && !((unsigned)x < (unsigned)pl.n[0] && (unsigned)y < (unsigned)pl.n[1] && (DIM == 2 || (unsigned)z < (unsigned)pl.n[2]))) return -1;
        return DIM == 3 ? ((b * pl.n[2] + z) * pl.n[1] + y) * pl.n[0] + x : (b * pl.n[1] + y) * pl.n[0] + x;
    };
    first = brick(kc);
    second = brick(kc + 1.f);
}
// The shift phase of a listed pixel, as phase_of_dot: the shifts of listed slices are small enough for the sum.
__device__ __forceinline__ float2 list_phase(const SliceGeom& g, float dot) {
    const float k = dot * g.inv_n + kRound - kRound, angle = fmaf(-k, g.n_f, dot) * g.phase_scale_f;
    return make_float2(__cosf(angle), __sinf(angle));
}
__device__ __forceinline__ bool list_has_slice(const ListWork& ws, int k) { return !isnan(__ldg(&ws.poses[2 * (size_t)k].x)); }

// How many of a brick's cells the pixels of a call share: pixels of slices drawn at random, the brick and the cell of each, and
// the pixels of another slice that lie in this brick (header[8]) and in this cell (header[9]).  Their ratio is the number of cells that
// would be as crowded if all were alike: 330-570 of 512 for uniform poses, poses about one axis with free in-plane turns, and within 15
// degrees of one view; 60 for slices of one plane (any turn), 15 for slices of one pose (oversampled twice: one sample in four
// cells of a plane), 45-70 for a tilt series (200 not oversampled), 90 for a hundred poses, 75 when half the slices share a plane.
__device__ __forceinline__ unsigned probe_bits(unsigned x) {            // (Wellons' "lowbias32" hash)
    x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
    return x;
}
template <int DIM>
__device__ __forceinline__ void list_probe(const float* __restrict__ rot, const ListWork& ws, const SliceGeom& g, const ListPlan& pl, int draw) {
    using L = ListBrick<DIM>;
    constexpr unsigned kFull = 0xffffffffu;
    constexpr int kHits = DIM == 3 ? 2 : 1, kFar = 16;         // hits of a warp that are counted; reach of the search, in pixels
    constexpr float kHalfX = 0.5f * (1 << L::kLogX), kHalfY = 0.5f * (1 << L::kLogY), kHalfZ = DIM == 3 ? 0.5f * (1 << L::kLogZ) : 0.f;
    constexpr float kDiagonal = DIM == 3 ? 6.94f : 11.33f;      // from the centre of a brick to its corners
    const int lane = threadIdx.x & 31, half = g.N / 2;
    auto columns = [&](int k, float4& ra, float4& rb) {
        const int b = k / g.P;
        const float* rm = pose_rot<DIM>(g, rot, b, k - b * g.P);
        ra = make_float4(__ldg(rm), __ldg(rm + DIM), DIM == 3 ? __ldg(rm + 6) : 0.f, __ldg(rm + 1));
        rb = make_float4(__ldg(rm + DIM + 1), DIM == 3 ? __ldg(rm + 7) : 0.f, 0.f, 0.f);
    };
    auto brick = [&](const ListSample& s) { return make_int3(s.x >> L::kLogX, s.y >> L::kLogY, DIM == 3 ? s.z >> L::kLogZ : 0); };
    auto listed = [&](int kr, int kc) { return kr > -half && kr <= half && kc >= 0 && kc <= half && (float)(kr * kr + kc * kc) <= g.cutoff_sq && !(kc == 0 && (kr < 0 || kr == half)); };
    const unsigned seed = 4u * (unsigned)draw;
    const int k = (int)__umulhi(probe_bits(seed), (unsigned)g.BP), first = k - k % g.P;
    int other = k + 1 + (int)__umulhi(probe_bits(seed + 1u), (unsigned)(g.P - 1));
    if (other >= first + g.P) other -= g.P;
    // a pixel within the cutoff, of those in the rows and columns that it reaches
    const float within = fminf((float)half, sqrtf(g.cutoff_sq));
    const int reach = (int)within, kr = (int)__umulhi(probe_bits(seed + 2u), 2u * (unsigned)reach + 1u) - reach, kc = (int)__umulhi(probe_bits(seed + 3u), (unsigned)reach + 1u);
    float4 ra, rb;
    columns(k, ra, rb);
    const ListSample s = list_sample<DIM>(g, pl, ra, rb, (unsigned)(kr + half - 1), (unsigned)kc);
    const int3 at = brick(s);
    bool hit = listed(kr, kc) && (unsigned)at.x < (unsigned)pl.n[0] && (unsigned)at.y < (unsigned)pl.n[1] && (DIM == 2 || (unsigned)at.z < (unsigned)pl.n[2]);
    // where the other slice comes closest to the centre of the brick: the least squares solution for its columns
    columns(other, ra, rb);
    const float x = (float)(at.x * (1 << L::kLogX) + pl.lo[0]) + kHalfX, y = (float)(at.y * (1 << L::kLogY) + pl.lo[1]) + kHalfY, z = DIM == 3 ? (float)(at.z * (1 << L::kLogZ) + pl.lo[2]) + kHalfZ : 0.f;
    const float aa = ra.x * ra.x + ra.y * ra.y + ra.z * ra.z, ab = ra.x * ra.w + ra.y * rb.x + ra.z * rb.y, bb = ra.w * ra.w + rb.x * rb.x + rb.y * rb.y;
    const float u = ra.x * x + ra.y * y + ra.z * z, v = ra.w * x + rb.x * y + rb.y * z, det = aa * bb - ab * ab;
    const float col = (bb * u - ab * v) / det, row = (aa * v - ab * u) / det, least = 0.5f * (aa + bb - sqrtf((aa - bb) * (aa - bb) + 4.f * ab * ab)),
                far = ceilf(kDiagonal * rsqrtf(least) / g.os_f + 0.5f);
    const float dx = ra.x * col + ra.w * row - x, dy = ra.y * col + rb.x * row - y, dz = ra.z * col + rb.y * row - z;
    hit = hit && det > 0.f && least > 0.f && far <= (float)kFar && dx * dx + dy * dy + dz * dz <= kDiagonal * kDiagonal;
    const int near_col = hit ? __float2int_rn(col / g.os_f) : 0, near_row = hit ? __float2int_rn(row / g.os_f) : 0, wide = hit ? 2 * (int)far + 1 : 0;
    int in_brick = 0, in_cell = 0;
    unsigned hits = __ballot_sync(kFull, hit);
    for (int q = 0; q < kHits && hits != 0u; ++q, hits &= hits - 1u) {
        const int from = __ffs(hits) - 1;
        const float4 fa = make_float4(__shfl_sync(kFull, ra.x, from), __shfl_sync(kFull, ra.y, from), __shfl_sync(kFull, ra.z, from), __shfl_sync(kFull, ra.w, from));
        const float4 fb = make_float4(__shfl_sync(kFull, rb.x, from), __shfl_sync(kFull, rb.y, from), 0.f, 0.f);
        const int w = __shfl_sync(kFull, wide, from), c0 = __shfl_sync(kFull, near_col, from) - w / 2, r0 = __shfl_sync(kFull, near_row, from) - w / 2;
        const int cx = __shfl_sync(kFull, s.x, from), cy = __shfl_sync(kFull, s.y, from), cz = __shfl_sync(kFull, s.z, from);
        for (int t = lane; t < w * w; t += 32) {
            // pixels of the half that is not stored are the conjugates of those at the opposite place, which were folded over
            int c = c0 + t % w, r = r0 + t / w;
            const bool opposite = c < 0;
            if (opposite) {
                c = -c;
                r = -r;
            }
            if (!listed(r, c)) continue;
            const ListSample o = list_sample<DIM>(g, pl, fa, fb, (unsigned)(r + half - 1), (unsigned)c);
            if (o.folded != opposite) continue;
            in_brick += o.x >> L::kLogX == cx >> L::kLogX && o.y >> L::kLogY == cy >> L::kLogY && (DIM == 2 || o.z >> L::kLogZ == cz >> L::kLogZ);
            in_cell += o.x == cx && o.y == cy && o.z == cz;
        }
    }
    in_brick = __reduce_add_sync(kFull, in_brick);
    in_cell = __reduce_add_sync(kFull, in_cell);
    if (lane == 0 && in_brick > 0) {
        atomicAdd(ws.header + 8, in_brick);
        if (in_cell > 0) atomicAdd(ws.header + 9, in_cell);
    }
}

// Blocks of 256 threads: one per 16 rows and 32 columns of a slice, one per 256 slices, then pl.probes.  The header is zero on entry.
// Pixels outside the cutoff and the mirrored half of column 0 are left out.  Slices with matrices or shifts that are not
// finite, or so large that the arithmetic above would not hold, are not listed.
template <int DIM>
__global__ void __launch_bounds__(256)
list_setup_kernel(const float* __restrict__ rot, const float* __restrict__ shifts, ListWork ws, const SliceGeom g, const ListPlan pl) {
    const int across = (g.Nh + 31) / 32, tiles = g.tiles_i * across, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if ((int)blockIdx.x < tiles) {
        // a warp: 4 rows of 8 pairs
        const int ti = (int)blockIdx.x / across, i = ti * 16 + (warp >> 1) * 4 + (lane >> 3), j = ((int)blockIdx.x - ti * across) * 32 + (warp & 1) * 16 + (lane & 7) * 2;
        const int row = i <= g.N / 2 ? i : i - g.N;
        const float kr = (float)row;
        auto listed = [&](int c) {
            const float kc = (float)c;
            return i < g.N && c < g.Nh && !(add_rn(mul_rn(kr, kr), mul_rn(kc, kc)) > g.cutoff_sq) && !(c == 0 && i >= g.N / 2);
        };
        const bool first = listed(j), second = listed(j + 1);
        const unsigned m = __ballot_sync(0xffffffffu, first || second);
        int at = 0;
        if (lane == 0 && m != 0u) at = atomicAdd(ws.header + 7, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (first || second)
            ws.inside[at + __popc(m & ((1u << lane) - 1u))] = (unsigned)(row + g.N / 2 - 1) << pl.bits_j | (unsigned)j | (first ? 0x40000000u : 0u) | (second ? 0x80000000u : 0u);
        return;
    }
    const int t = ((int)blockIdx.x - tiles) * 256 + (int)threadIdx.x;
    if ((int)blockIdx.x - tiles >= (g.BP + 255) / 256) {
        list_probe<DIM>(rot, ws, g, pl, t);
        return;
    }
    if (t >= g.BP) return;
    const int b = t / g.P, p = t - b * g.P;
    const float* rm = pose_rot<DIM>(g, rot, b, p);
    const float2 s = g.has_shift ? make_float2(__ldg(pose_shift(g, shifts, b, p)), __ldg(pose_shift(g, shifts, b, p) + 1)) : make_float2(0.f, 0.f);
    float4 ra = make_float4(__ldg(rm), __ldg(rm + DIM), DIM == 3 ? __ldg(rm + 6) : 0.f, __ldg(rm + 1));
    const float4 rb = make_float4(__ldg(rm + DIM + 1), DIM == 3 ? __ldg(rm + 7) : 0.f, s.x, s.y);
    if (!(fmaxf(fmaxf(fabsf(ra.x), fabsf(ra.y)), fmaxf(fabsf(ra.z), fabsf(ra.w))) < 1e30f && fmaxf(fabsf(rb.x), fabsf(rb.y)) < 1e30f &&
          fmaxf(fabsf(s.x), fabsf(s.y)) < 1e5f) || isnan(ra.x + ra.y + ra.z + ra.w + rb.x + rb.y + s.x + s.y)) {
        ra.x = __int_as_float(0x7fffffff);
        atomicAdd(ws.header + 4, 1);
    } else if (!(pl.reach * sqrtf(ra.x * ra.x + ra.w * ra.w) <= pl.fit[0] && pl.reach * sqrtf(ra.y * ra.y + rb.x * rb.x) <= pl.fit[1] &&
                 (DIM == 2 || pl.reach * sqrtf(ra.z * ra.z + rb.y * rb.y) <= pl.fit[2]))) {
        atomicAdd(ws.header + 6, 1);
    }
    ws.poses[2 * (size_t)t] = ra;
    ws.poses[2 * (size_t)t + 1] = rb;
}

// Where the counter of a brick lies: groups of eight bricks (a sector of L2) are spread over the lines.  One after the other, the
// counters of a plane's bricks share a few dozen lines, where atomics queue up.
__device__ __forceinline__ unsigned list_counter(const ListPlan& pl, int brick) {
    return ((((unsigned)brick >> 3) * pl.spread) & pl.groups) << 3 | ((unsigned)brick & 7u);
}

constexpr int kListRun = 2;                 // pairs of pixels of a thread at a time
constexpr int kListPairs = 256 * kListRun;  // of a block
constexpr int kListBricks = 4096;           // bricks of a batch item that a block can count in shared memory

// A lane takes a pair of pixels of a row.  The lanes of a warp whose first pixels lie in the same brick send one atomic
// between them, in which second pixels join that lie in the brick of their own first pixel or of the next lane's; the few
// others go by themselves.  (The match instruction holds the SM's only unit for it for 31 clocks: with one per 32 pixels, not per
// 64, a pass took 3.5 ps per pixel.)
//   pl.run == 0: counts in global memory, pl.subs for each brick, which slices use in turn: atomics at the bricks that many slices meet
//   in would queue up.  But each is a place where the second pass writes, and beyond some 40,000 such places sectors leave L2
//   half written.  (Passes in us with 1 / 4 / 8 / 16 counters, all one after the other: 2,501 slices of 90 x 46, 3,000 bricks met, 49 + 55 / 26 + 36 /
//   26 + 36 / 26 + 36; 50,000 of 128 x 65, 8,600 bricks, 1,070 + 1,500 / 886 + 1,444 / 892 + 1,545 / 892 + 1,670; 4,096 of 256 x 129, 68,000 bricks,
//   280 + 472 / 261 + 582 / 262 + 648 / 261 + 725.)  In groups spread over the lines (list_counter), four of them: 10,000 slices of 128 x 65 in one
//   plane 812 + 852 -> 161 + 255, within 15 degrees of one view 324 + 391 -> 162 + 237, of uniform poses 173 + 272 -> 165 + 251.
//   Grid: x = kListPairs pairs of a slice, y = pl.turn slices, one after the other.
//   else: bricks are few and many slices meet in each (2D: all slices in every tile), so atomics would queue up at a few
//   addresses.  A block counts pl.run slices of a batch item in shared memory, and keeps its counts for the second pass.
//   Grid: x = runs of a batch item, y = batch item.
// (1,000 slices of 128 x 65 onto each of eight 256 x 129 references: 1,750 us a pass in global memory, 120 in shared memory.)
template <int DIM, bool COUNT, bool SHARED>
__global__ void __launch_bounds__(256, 6)
list_pixels_kernel(ListWork ws, const SliceGeom g, const ListPlan pl) {
    __shared__ unsigned here[SHARED ? kListBricks : 1];
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31, tid = threadIdx.x;
    const unsigned below = (1u << lane) - 1u;
    if (Gate::crowded(ws.header, pl.crowd)) return;
    const bool all_fit = __ldg(ws.header + 6) == 0;
    int slice, last, begin = 0, end = __ldg(ws.header + 7), b = 0;
    unsigned* row = nullptr;
    if (SHARED) {
        // runs do not cross batch items
        b = (int)blockIdx.y;
        slice = max(b * g.P, pl.first) + (int)blockIdx.x * pl.run - pl.first;
        last = min(min((b + 1) * g.P, pl.first + pl.slices) - pl.first, slice + pl.run);
        if (slice >= last) return;
        row = ws.block_count + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * (size_t)pl.item_bricks;
        for (int t = tid; t < pl.item_bricks; t += 256) {
            unsigned n = 0u;
            if (!COUNT) {
                n = row[t];
                if (n != 0u) n = atomicAdd(ws.count + list_counter(pl, b * pl.item_bricks + t), n);
            }
            here[t] = n;
        }
        __syncthreads();
    } else {
        slice = ((int)blockIdx.y + (int)blockIdx.z * 32768) * pl.turn;
        last = min(pl.slices, slice + pl.turn);
        begin = (int)blockIdx.x * kListPairs;
        end = min(end, begin + kListPairs);
    }
    for (; slice < last; ++slice) {
        const int k = pl.first + slice;
        if (!SHARED) b = k / g.P;
        const float4 ra = __ldg(ws.poses + 2 * (size_t)k), rb = __ldg(ws.poses + 2 * (size_t)k + 1);
        if (isnan(ra.x)) continue;
        for (int base = begin; base < end; base += kListPairs) {
            unsigned entry[kListRun], same[kListRun], own[kListRun], next[kListRun], at[kListRun], at2[kListRun];
            int brick[kListRun], brick2[kListRun];
#pragma unroll
            for (int q = 0; q < kListRun; ++q) {
                const int t = base + q * 256 + tid;
                const unsigned pair = t < end ? __ldg(ws.inside + t) : 0u;
                entry[q] = pair & 0x3fffffffu;
                list_bricks<DIM>(g, pl, ra, rb, entry[q], SHARED ? 0 : b, all_fit, brick[q], brick2[q]);
                if ((pair & 0x40000000u) == 0u) brick[q] = -1;
                if ((pair & 0x80000000u) == 0u) brick2[q] = -1;
            }
#pragma unroll
            for (int q = 0; q < kListRun; ++q) {
                same[q] = __match_any_sync(kFull, brick[q]);
                const int right = __shfl_down_sync(kFull, brick[q], 1);
                const bool to_own = brick2[q] >= 0 && brick2[q] == brick[q], to_next = brick2[q] >= 0 && !to_own && lane < 31 && brick2[q] == right;
                own[q] = __ballot_sync(kFull, to_own);
                next[q] = __ballot_sync(kFull, to_next) << 1;       // by the lane whose brick it is
                at[q] = at2[q] = 0u;
                unsigned* counts = SHARED ? here : ws.count + (size_t)(slice & (pl.subs - 1)) * (size_t)(8u * (pl.groups + 1u));
                if (brick[q] >= 0 && (same[q] & below) == 0u) {
                    const unsigned n = __popc(same[q]) + __popc(same[q] & own[q]) + __popc(same[q] & next[q]);
                    unsigned* c = counts + (SHARED ? (unsigned)brick[q] : list_counter(pl, brick[q]));
                    if (COUNT) atomicAdd(c, n);
                    else at[q] = atomicAdd(c, n);
                }
                if (brick2[q] >= 0 && !to_own && !to_next) {
                    unsigned* c = counts + (SHARED ? (unsigned)brick2[q] : list_counter(pl, brick2[q]));
                    if (COUNT) atomicAdd(c, 1u);
                    else at2[q] = atomicAdd(c, 1u);
                }
            }
            if (COUNT) continue;
#pragma unroll
            for (int q = 0; q < kListRun; ++q) {
                // first pixels, then the second ones of the same lanes, then those of the lanes to the left
                const unsigned first = __shfl_sync(kFull, at[q], max(__ffs(same[q]) - 1, 0)), all = same[q];
                const unsigned first_r = __shfl_down_sync(kFull, first, 1), all_r = __shfl_down_sync(kFull, all, 1);
                const unsigned e = (unsigned)slice << (pl.bits_i + pl.bits_j) | entry[q];
                const unsigned to = first + __popc(all & below);
                if (brick[q] >= 0 && to < pl.capacity) ws.list[to] = e;
                unsigned to2 = at2[q];
                if (own[q] >> lane & 1u) to2 = first + __popc(all) + __popc(all & own[q] & below);
                else if (lane < 31 && (next[q] >> (lane + 1) & 1u)) to2 = first_r + __popc(all_r) + __popc(all_r & own[q]) + __popc(all_r & next[q] & ((2u << lane) - 1u));
                if (brick2[q] >= 0 && to2 < pl.capacity) ws.list[to2] = e + 1u;
            }
        }
    }
    if (SHARED && COUNT) {
        __syncthreads();
        for (int t = tid; t < pl.item_bricks; t += 256) {
            const unsigned n = here[t];
            row[t] = n;
            if (n != 0u) atomicAdd(ws.count + list_counter(pl, b * pl.item_bricks + t), n);
        }
    }
}

// A place in the list and work items for each brick.  Bricks are taken along a Morton curve, so that neighbours run at the
// same time: they read the same sectors of the slices.
template <int DIM>
__global__ void __launch_bounds__(256)
list_plan_kernel(ListWork ws, const ListPlan pl, int B) {
    if (Gate::crowded(ws.header, pl.crowd)) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned t = blockIdx.x * 256u + threadIdx.x, place = t & ((1u << (DIM * pl.bits)) - 1u);
    const int b = (int)(t >> (DIM * pl.bits));
    int x = 0, y = 0, z = 0;
    for (int k = 0; k < pl.bits; ++k) {
        x |= (int)(place >> (DIM * k) & 1u) << k;
        y |= (int)(place >> (DIM * k + 1) & 1u) << k;
        if (DIM == 3) z |= (int)(place >> (DIM * k + 2) & 1u) << k;
    }
    const bool here = b < B && x < pl.n[0] && y < pl.n[1] && z < pl.n[2];
    const int brick = ((b * pl.n[2] + z) * pl.n[1] + y) * pl.n[0] + x;
    const unsigned counter = list_counter(pl, brick);
    int n = 0;
    if (here)
        for (int k = 0; k < pl.subs; ++k) n += (int)ws.count[(size_t)k * (size_t)(8u * (pl.groups + 1u)) + counter];
    const int parts = (n + pl.most - 1) / pl.most;
    int n_upto = n, parts_upto = parts;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, n_upto, o), c = __shfl_up_sync(0xffffffffu, parts_upto, o);
        if (lane >= o) {
            n_upto += a;
            parts_upto += c;
        }
    }
    __shared__ int warp_n[8], warp_parts[8], base[2];
    if (lane == 31) {
        warp_n[warp] = n_upto;
        warp_parts[warp] = parts_upto;
    }
    if (__syncthreads_or(n) == 0) return;
    if (threadIdx.x < 2) {
        int* w = threadIdx.x == 0 ? warp_n : warp_parts;
        int sum = 0;
        for (int k = 0; k < 8; ++k) { const int m = w[k]; w[k] = sum; sum += m; }
        base[threadIdx.x] = sum > 0 ? atomicAdd(ws.header + threadIdx.x, sum) : 0;
    }
    __syncthreads();
    const int first = base[0] + warp_n[warp] + n_upto - n;
    if (n > 0) {
        int at = first;
        for (int k = 0; k < pl.subs; ++k) {
            unsigned& c = ws.count[(size_t)k * (size_t)(8u * (pl.groups + 1u)) + counter];
            const int m = (int)c;
            c = (unsigned)at;
            at += m;
        }
    }
    // Items part by part: the first of all bricks of the block, then the second ...  Neighbours then go through the same
    // slices at the same time, whose sectors they share.
    __shared__ int level[2][8];
    const int share = n / max(parts, 1), more = n - share * parts;
    int place_at = base[1];
    for (int q = 0;; ++q) {
        const unsigned m = __ballot_sync(0xffffffffu, parts > q);
        if (lane == 0) level[q & 1][warp] = __popc(m);
        if (__syncthreads_or(parts > q) == 0) break;
        int before = 0, all = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            const int c = level[q & 1][w];
            before += w < warp ? c : 0;
            all += c;
        }
        if (parts > q) ws.items[place_at + before + __popc(m & ((1u << lane) - 1u))] = make_int4(brick, first + q * share + min(q, more), share + (q < more ? 1 : 0), 0);
        place_at += all;
    }
}

}  // namespace b200proj
