// mdx_segm.cuh -- segmented (batched) stable m-way partition for sm_100a.
//
// Replaces mdiscrSegm<DISCR> (cuda_code/MdiscrSegmHost.cu.h:36-230: a chain
// of ~12 kernels -- segmented scans of head flags and of N one-hot m-tuples,
// per-element reductions, class offsets, indices, permute, sizes -- with nine
// N-sized temporaries, four of them N*m tuples) by six launches:
//
//   seg_plan_spans  per segment: its length.  Segments longer than one tile
//                   (P elements) are "large" and are cut into runs of up to
//                   RUN_TILES tiles; the other ("small") segments are grouped
//                   (consecutive small segments starting in one window of
//                   P elements, at most kGroupSegs of them).  Block-local
//                   scans of the run and group counts; the last CTA scans the
//                   block totals, records the counts and resets the tickets.
//   seg_plan_emit   writes the run entries {segment, [p0, p1), last run of
//                   the segment} and the group heads, in element order.
//   seg_main        persistent; CTAs take tickets for batches of groups.  A
//                   group's range is read into shared memory by one bulk copy and
//                   partitioned by the whole CTA (seg_group_cta: every thread owns
//                   consecutive elements whatever the segment lengths; one scan of
//                   per-thread class counts gives every segment's sizes and every
//                   element's place) into a shared output image that one bulk store
//                   writes back -- one HBM read and one write per element;
//   seg_run_count   the class counts of every run of the large segments, one CTA per
//                   run (16-byte loads, warp reductions);
//   seg_run_scan    per large segment (a lane, or a warp for many runs):
//                   the runs' exclusive class prefixes, the segment's sizes
//                   and head flags, and every run's output position per class.
//   seg_run_scatter persistent; the runs in reverse order through a TMA ring
//                   and tile_scatter (as the plain scatter), from those
//                   positions.
//
// The partition kernels and the head-flag converter wait on no other CTA, only
// on their own bulk copies.
// Every wait is bounded by kWaitLimitNs; one that runs out latches
// kErrTimeout and publishes what it has, so no other CTA waits forever.
//
// Output per segment equals seqMdiscr (SeqMdiscr.h:10-57) applied to the
// segment, which is exactly what MdiscrSegmTest.cu:8-41 validates; sizes are
// emitted as an S x m tuple table and/or per-segment head flags
// (MdiscrSegmKernels.cu.h:89-114 writes the latter into new_sizes).
#pragma once

#include <cuda.h>  // CUtensorMap

#include <type_traits>

#include "mdx_device.cuh"
#include "mdx_plain.cuh"  // PackedCounts
#include "mdx_tile.cuh"

namespace mdx {

// Defaults of the run-time knobs (the autotuner may choose others):
constexpr int kRunTiles = 8;     // tiles per run of a large segment
constexpr int kMidTiles = 2;     // most tiles a medium segment may span (seg_mid's slab)
constexpr int kGroupBatch = 8;   // small-segment groups per ticket of seg_main
constexpr int kMaxGroupBatch = 32;
constexpr uint32_t kMaxPlanBlocks = 1024;

struct SegHeader {      // lives at the start of the segmented workspace
    uint32_t ticket;    // seg_main's tickets (reset by the planner)
    uint32_t error;     // latched error bits
    uint32_t num_mids;  // medium segments this call
    uint32_t num_runs;  // large-segment runs this call
    uint32_t ticket4;   // seg_mid's segment tickets (reset by the planner)
    uint32_t plan_done; // planner CTA ticket
    uint64_t num_segs;  // S (written by the flags converter for the head-flag form)
    uint32_t reserved2;
    uint32_t reserved3;
    uint32_t flags_done;    // finished chunks of the flags converter (reset by its last CTA)
    uint32_t reserved4;
    uint32_t num_groups;    // small-segment groups this call
    uint32_t ticket2;       // run-scatter ticket counter (reset by the planner)
    uint32_t ticket3;       // run-count ticket counter (reset by the planner)
    uint32_t pad[1];
};

struct alignas(16) RunEntry {  // a run of up to run_tiles tiles of one large segment
    uint32_t seg;              // segment index
    uint32_t p0;               // its first element
    uint32_t len_m;            // its length (low 24 bits: at most 64 tiles) and, when the call
                               // carries class counts per segment, the segment's (high 8)
    uint32_t jlast;            // entry index of the segment's last run
    __device__ __forceinline__ uint32_t p1() const { return p0 + (len_m & 0xffffffu); }
};

struct SegArgs {
    const void* in;
    void* out;
    uint64_t n;
    const uint64_t* offsets;   // S+1
    uint64_t num_segs;         // S, or kSegsOnDevice: read hdr->num_segs
    uint32_t* seg_sizes;       // S*m or null
    uint32_t* headflags;       // n or null (zeroed before the main kernel)
    const int32_t* in_flags;   // head-flag input (validated by the planner) or null
    uint32_t m;
    SegHeader* hdr;
    uint32_t* run_loc;         // [S] block-local exclusive run offsets
    uint32_t* grp_loc;         // [S] block-local exclusive group-head offsets
    uint32_t* blk_runs;        // [plan blocks] run totals, then offsets
    uint32_t* blk_grps;        // [plan blocks] group totals, then offsets
    RunEntry* runs;            // [max_runs]
    uint32_t* groups;          // [max_groups] first segment of each group
    uint32_t* groups_end;      // [max_groups] one past its last segment (0xffffffff: none
                               // marked, the group runs to S; reset every call)
    uint32_t* run_cnt;         // [max_runs][M] class counts of each run
    uint32_t* run_base;        // [max_runs][M] output position of each run's first element per class
    uint32_t plan_blocks;
    uint32_t max_runs;         // capacity (enough for segments that tile [0, n))
    uint32_t max_groups;
    int use_tma;               // the tensor map passed to seg_run_scatter is valid
    const uint32_t* seg_m;     // per-segment class counts (remainder discriminator), or null:
                               // every segment uses the launch's discriminator
    uint32_t m_bound;          // classes of any segment are < m_bound (per-segment m clamped)
    uint32_t run_tiles;        // tiles per run of a large segment
    uint32_t group_batch;      // small-segment groups per work item
    uint32_t mid_tiles;        // a segment of more than one tile that spans at most this
                               // many row-aligned tiles is medium (0: none are)
    uint32_t* mid_loc;         // [S] block-local exclusive medium-segment offsets
    uint32_t* blk_mids;        // [plan blocks] medium-segment totals, then offsets
    uint32_t* mids;            // [max_mids] the medium segments, in order
    uint32_t max_mids;
};

// Class count of segment s, clamped to [1, m_bound], when the call carries them.
__device__ __forceinline__ uint32_t seg_classes(const SegArgs& a, uint64_t s) {
    return a.seg_m != nullptr ? min(max(a.seg_m[s], 1u), a.m_bound) : 0u;
}
// The discriminator of a segment with class count m: the launch's, or -- when the
// call carries class counts per segment -- key % m.
template <class D>
__device__ __forceinline__ D seg_discr(const SegArgs& a, const D& d, uint32_t m) {
    if constexpr (std::is_same<D, DiscrMod>::value) {
        if (a.seg_m != nullptr) return DiscrMod::make(m);
    }
    return d;
}

constexpr uint64_t kSegsOnDevice = ~0ull;

// Small segments are grouped: a group is a run of consecutive small segments
// whose first elements lie in one window of P elements, cut after at most
// kGroupSegs segments, so a group spans < 2P elements.
constexpr uint32_t kGroupSegs = 128;
template <int P>
__host__ __device__ constexpr uint64_t group_window() {
    return static_cast<uint64_t>(P);
}
template <int P>
__device__ __forceinline__ bool group_head(const SegArgs& a, uint64_t s, uint64_t a0) {
    constexpr uint64_t GW = group_window<P>();
    return s == 0 || a.offsets[s - 1] / GW != a0 / GW || (s % kGroupSegs) == 0;
}

// A segment's tiles start at the 128-byte row holding its first element (a
// tile is P * sizeof(V) = 16 KB, so a row is P / 128 elements): the TMA box
// needs a row start, and tiles counted from there leave only the last one
// short.
template <int P>
__device__ __forceinline__ uint64_t seg_row_start(uint64_t a0) {
    return a0 & ~(static_cast<uint64_t>(P) / 128u - 1u);
}
template <int P>
__device__ __forceinline__ uint32_t seg_tiles(uint64_t a0, uint64_t a1) {
    return static_cast<uint32_t>((a1 - seg_row_start<P>(a0) + P - 1u) / P);
}

// A segment [a0, a1) longer than one tile is medium when its tiles number at
// most mid_tiles: seg_mid then reads it once.  The longer ones are cut into
// runs of run_tiles of those tiles (every run but the last is whole tiles).
template <int P>
__device__ __forceinline__ bool is_mid(const SegArgs& a, uint64_t a0, uint64_t a1) {
    return a.mid_tiles > 0u && seg_tiles<P>(a0, a1) <= a.mid_tiles;
}

__device__ __forceinline__ uint64_t seg_count(const SegArgs& a) {
    return a.num_segs == kSegsOnDevice ? a.hdr->num_segs : a.num_segs;
}

// Whether segment s of S, [a0, a1), can be one of the segments that tile [0, n).  Both
// planning kernels leave the others alone, by this one test: entries of a segment that
// was given no room would take another's, and runs of two segments mixed under one
// can reach past its end.
__device__ __forceinline__ bool seg_in_place(const SegArgs& a, uint64_t s, uint64_t S, uint64_t a0,
                                             uint64_t a1) {
    return a0 <= a1 && a1 <= a.n && (s != 0 || a0 == 0) && (s + 1 != S || a1 == a.n);
}

// --------------------------------------------------------------- planning --
// Block b of the planner owns segments [b*R, min((b+1)*R, S)), R = ceil(S/G).
template <int P, int THREADS>
__global__ void __launch_bounds__(THREADS) seg_plan_spans(SegArgs a) {
    constexpr int W = THREADS / 32;
    __shared__ uint32_t warp_runs[W], warp_grps[W], warp_mids[W];
    __shared__ int am_last;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_launch_dependents();
    const uint64_t S = seg_count(a);
    // no group has an end yet
    for (uint32_t g = blockIdx.x * THREADS + tid; g < a.max_groups; g += gridDim.x * THREADS)
        a.groups_end[g] = 0xffffffffu;
    const uint64_t G = gridDim.x;
    const uint64_t R = (S + G - 1) / G;
    const uint64_t s0 = blockIdx.x * R, s1 = min(s0 + R, S);
    uint32_t carry_r = 0, carry_g = 0, carry_m = 0;
    for (uint64_t base = s0; base < s1; base += THREADS) {
        const uint64_t s = base + tid;
        uint32_t runs = 0, head = 0, mid = 0;
        if (s < s1) {
            const uint64_t a0 = a.offsets[s], a1 = a.offsets[s + 1];
            if (!seg_in_place(a, s, S, a0, a1)) {
                atomicOr(&a.hdr->error, kErrSegments);
            } else if (a1 - a0 > static_cast<uint64_t>(P)) {
                if (is_mid<P>(a, a0, a1)) {
                    mid = 1;
                } else {
                    runs = (seg_tiles<P>(a0, a1) + a.run_tiles - 1) / a.run_tiles;
                }
            } else {
                head = group_head<P>(a, s, a0) ? 1u : 0u;
            }
            if (a.in_flags != nullptr && a1 > a0 && a1 <= a.n &&
                static_cast<uint64_t>(a.in_flags[a0]) != a1 - a0)
                atomicOr(&a.hdr->error, kErrSegments);
            if (a.seg_m != nullptr && (a.seg_m[s] < 1u || a.seg_m[s] > a.m_bound))
                atomicOr(&a.hdr->error, kErrSegments);
        }
        const uint32_t ir = warp_incl_scan(runs);
        const uint32_t ig = warp_incl_scan(head);
        const uint32_t im = warp_incl_scan(mid);
        if (lane == 31) {
            warp_runs[warp] = ir;
            warp_grps[warp] = ig;
            warp_mids[warp] = im;
        }
        __syncthreads();
        uint32_t pr = 0, pg = 0, pm = 0, tr = 0, tg = 0, tm = 0;
        for (int w = 0; w < W; w++) {
            const uint32_t xr = warp_runs[w], xg = warp_grps[w], xm = warp_mids[w];
            pr += (w < warp) ? xr : 0u;
            pg += (w < warp) ? xg : 0u;
            pm += (w < warp) ? xm : 0u;
            tr += xr;
            tg += xg;
            tm += xm;
        }
        if (s < s1) {
            a.run_loc[s] = carry_r + pr + ir - runs;
            a.grp_loc[s] = carry_g + pg + ig - head;
            a.mid_loc[s] = carry_m + pm + im - mid;
        }
        // segments that overlap can have more runs than 32 bits count: one more than
        // there is room for says as much (groups and medium segments are at most S)
        carry_r = min(carry_r + tr, a.max_runs + 1u);
        carry_g += tg;
        carry_m += tm;
        __syncthreads();
    }
    if (tid == 0) {
        a.blk_runs[blockIdx.x] = carry_r;
        a.blk_grps[blockIdx.x] = carry_g;
        a.blk_mids[blockIdx.x] = carry_m;
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) am_last = (atomicAdd(&a.hdr->plan_done, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!am_last) return;
    __threadfence();
    // last CTA: exclusive scans of the block totals (in place), four a thread so that
    // all are in flight at once
    static_assert(4 * THREADS >= kMaxPlanBlocks, "four block totals a thread");
    uint32_t* const arrs[3] = {a.blk_runs, a.blk_grps, a.blk_mids};
    const uint32_t bounds[3] = {a.max_runs, a.max_groups, a.max_mids};
    uint32_t* const counts[3] = {&a.hdr->num_runs, &a.hdr->num_groups, &a.hdr->num_mids};
    uint32_t* const wsum[3] = {warp_runs, warp_grps, warp_mids};
    uint32_t x[3][4], incl[3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint32_t b = 4u * tid + u;
            x[q][u] = b < gridDim.x ? __ldcg(&arrs[q][b]) : 0u;
        }
    }
#pragma unroll
    for (int q = 0; q < 3; q++) {
        incl[q] = warp_incl_scan(x[q][0] + x[q][1] + x[q][2] + x[q][3]);
        if (lane == 31) wsum[q][warp] = incl[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 3; q++) {
        uint32_t before = 0;
        uint64_t all = 0;
#pragma unroll
        for (int w = 0; w < W; w++) {
            before += w < warp ? wsum[q][w] : 0u;
            all += wsum[q][w];
        }
        uint32_t run = before + incl[q] - (x[q][0] + x[q][1] + x[q][2] + x[q][3]);
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (4u * tid + u < gridDim.x) arrs[q][4u * tid + u] = run;
            run += x[q][u];
        }
        if (tid == 0)  // over capacity: malformed
            *counts[q] = all <= bounds[q] ? static_cast<uint32_t>(all) : 0u;
    }
    __syncthreads();
    if (tid == 0) {
        a.hdr->ticket = 0u;
        a.hdr->ticket2 = 0u;
        a.hdr->ticket3 = 0u;
        a.hdr->ticket4 = 0u;
        a.hdr->plan_done = 0u;
    }
}

template <int P, int THREADS>
__global__ void __launch_bounds__(THREADS) seg_plan_emit(SegArgs a) {
    __shared__ uint32_t list_seg[THREADS], list_pos[THREADS], list_a0[THREADS], list_a1[THREADS];
    __shared__ uint32_t list_m[THREADS];
    __shared__ uint32_t list_n;
    const int tid = threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    const uint64_t S = seg_count(a);
    const uint64_t G = gridDim.x;
    const uint64_t R = (S + G - 1) / G;
    const uint64_t s0 = blockIdx.x * R, s1 = min(s0 + R, S);
    const uint32_t roff = a.blk_runs[blockIdx.x], goff = a.blk_grps[blockIdx.x];
    const uint32_t moff = a.blk_mids[blockIdx.x];
    const uint32_t num_runs = a.hdr->num_runs, num_groups = a.hdr->num_groups;
    const uint32_t num_mids = a.hdr->num_mids;
    // run r of the nr runs of segment s ([a0, a1), class count m), entries from pos on
    auto emit = [&](uint32_t s, uint32_t a0, uint32_t a1, uint32_t m, uint32_t pos, uint32_t nr,
                    uint32_t r) {
        const uint64_t rb = seg_row_start<P>(a0);
        const uint64_t len = static_cast<uint64_t>(a.run_tiles) * P;
        RunEntry e;
        e.seg = s;
        e.p0 = static_cast<uint32_t>(max(static_cast<uint64_t>(a0), rb + r * len));
        e.len_m = (static_cast<uint32_t>(min(static_cast<uint64_t>(a1), rb + (r + 1) * len)) - e.p0) |
                  (m << 24);
        e.jlast = pos + nr - 1u;
        a.runs[pos + r] = e;
    };
    for (uint64_t base = s0; base < s1; base += THREADS) {
        if (tid == 0) list_n = 0;
        __syncthreads();
        const uint64_t s = base + tid;
        if (s < s1) {
            const uint64_t a0 = a.offsets[s], a1 = a.offsets[s + 1];
            const bool in_place = seg_in_place(a, s, S, a0, a1);
            if (in_place) {
                if (a1 - a0 > static_cast<uint64_t>(P) && is_mid<P>(a, a0, a1)) {
                    const uint32_t pos = moff + a.mid_loc[s];
                    if (pos < num_mids) a.mids[pos] = static_cast<uint32_t>(s);
                } else if (a1 - a0 > static_cast<uint64_t>(P)) {
                    const uint32_t nr = (seg_tiles<P>(a0, a1) + a.run_tiles - 1) / a.run_tiles;
                    const uint32_t pos = roff + a.run_loc[s];
                    if (static_cast<uint64_t>(pos) + nr <= num_runs) {  // else malformed offsets
                        const uint32_t m = seg_classes(a, s);
                        if (nr <= 4) {  // this thread emits the runs itself
                            for (uint32_t r = 0; r < nr; r++)
                                emit(static_cast<uint32_t>(s), static_cast<uint32_t>(a0),
                                     static_cast<uint32_t>(a1), m, pos, nr, r);
                        } else {  // longer segments: a warp each, below
                            const uint32_t q = atomicAdd(&list_n, 1u);
                            list_seg[q] = static_cast<uint32_t>(s);
                            list_pos[q] = pos;
                            list_a0[q] = static_cast<uint32_t>(a0);
                            list_a1[q] = static_cast<uint32_t>(a1);
                            list_m[q] = m;
                        }
                    }
                } else if (group_head<P>(a, s, a0)) {
                    const uint32_t g = goff + a.grp_loc[s];
                    if (g < num_groups) a.groups[g] = static_cast<uint32_t>(s);
                }
            }
            // the group before segment s ends at s at the latest when s starts
            // a group, is large or is malformed
            const bool small_ok = in_place && a1 - a0 <= static_cast<uint64_t>(P);
            const bool is_head = small_ok && group_head<P>(a, s, a0);
            const uint32_t before = goff + a.grp_loc[s];  // groups starting before s
            if ((is_head || !small_ok) && before >= 1u && before - 1u < num_groups)
                atomicMin(&a.groups_end[before - 1u], static_cast<uint32_t>(s));
        }
        __syncthreads();
        const uint32_t cnt = list_n;
        for (uint32_t q = tid >> 5; q < cnt; q += THREADS / 32) {
            const uint32_t a0 = list_a0[q], a1 = list_a1[q];
            const uint32_t nr = (seg_tiles<P>(a0, a1) + a.run_tiles - 1) / a.run_tiles;
            for (uint32_t r = tid & 31; r < nr; r += 32)
                emit(list_seg[q], a0, a1, list_m[q], list_pos[q], nr, r);
        }
        __syncthreads();
    }
}

// --------------------------------------------------------------- main kernel --
template <int M, int THREADS>
struct GroupScratch;
template <int M, int THREADS>
constexpr size_t group_scratch_bytes();

template <class V, int M, int THREADS>
struct SegSmem {
    using G = TileGeom<V, THREADS, M>;
    static constexpr int kTile = G::kTile;  // == P
    static constexpr uint32_t kAU = G::kAU;
    // small groups (segments starting in one window of P, each <= P): an
    // input buffer and an output image, each for a range of < 2P elements plus
    // 16-byte alignment slack (the next group's copy overlaps the current
    // group's write-out; the other resident CTAs cover the rest of its latency)
    // A group's range is shorter than 2P.  Above 8 classes the scratch leaves three CTAs
    // to an SM buffers of 7/4 P: a longer group gives up its last segment to a group of
    // its own (both parts lie within P).  With buffers of 2P and two CTAs, groups of many
    // short segments, which latency bounds, were slower than before the class counts
    // were scanned without flags: 3 * 10^7 u32 in segments of 2 and of up to 32, m = 16,
    // a call 2855 and 1155 us, 2126 and 820 now (2103 and 899 with flags); log-normal
    // with median 1024, through head flags, 240 and 219; 2^20 elements in segments of
    // 4000, whose groups are all cut, 24 and 27.
    static constexpr int kGroupMost = M > 8 ? kTile / 4 * 7 : static_cast<int>(group_window<kTile>()) + kTile;
    static constexpr int kGroupElems = kGroupMost + 2 * static_cast<int>(kAU);
    static constexpr size_t kGroupBytes = 2ull * kGroupElems * sizeof(V);
    static constexpr size_t kBytes = 128 + kGroupBytes + group_scratch_bytes<M, THREADS>();  // seg_main
    static constexpr size_t kSmBytes = 228 * 1024, kReserved = 1024 + 128;  // of an SM, of a CTA
};

// seg_run_scatter: TMA slot + tile stage + count matrix
template <class V, int M, int THREADS>
struct RunSmem {
    using G = TileGeom<V, THREADS, M>;
    static constexpr size_t kSlotBytes = static_cast<size_t>(G::kTile) * sizeof(V);
    static constexpr size_t kBytes = 1024 + kSlotBytes + G::kStageBytes + G::kCntBytes;
};

// ------------------------------------------------------------ small segments --
// Shared state of one group (at most kGroupSegs segments).  Positions y count from
// the 16-byte address at or before the group's first element, in the input buffer
// and in the output image alike.
template <int M, int THREADS>
struct GroupScratch {
    static constexpr int NB = M > 4 ? M / 4 : 1;  // words of byte counts
    static constexpr int NH = M / 2;              // words of 16-bit counts
    // per segment, N words each (load, store)
    alignas(16) uint32_t hcnt[NB * kGroupSegs];  // its owner thread's class counts before the head
    alignas(16) uint32_t hpre[NH * kGroupSegs];  // the group's class counts before the head
    alignas(16) uint32_t hcur[NH * kGroupSegs];  // first position of each class of the segment
    uint32_t col[NH][THREADS];         // class counts before each thread's elements; before
                                       // that byte counters (M = 16), after it cursors (M > 4)
    uint32_t wagg[NH][THREADS / 32];
    uint16_t hpos[kGroupSegs + 2];     // head of each segment; [nseg] = the group's end
    uint8_t msz[kGroupSegs];           // the segment's class count (per-segment m)
    // Above 8 classes in 16-byte words, the two of eight u32 swapped in every other four
    // segments, so that neighbouring segments' words lie in different banks (3 * 10^7
    // u32 in segments of two and of up to 32, m = 16: 2185 and 895 us a call with every
    // word of its own, [word][segment], 2126 and 820 so).
    template <int N>
    static __device__ __forceinline__ uint32_t word(uint32_t seg, int q) {
        return N == 8 ? 2u * seg + (q ^ (seg >> 2 & 1u)) : N / 4 * seg + q;
    }
    template <int N>
    static __device__ __forceinline__ void load(const uint32_t* a, uint32_t seg, uint32_t (&x)[N]) {
        if constexpr (M > 8) {
#pragma unroll
            for (int q = 0; q < N / 4; q++) {
                const uint4 v = reinterpret_cast<const uint4*>(a)[word<N>(seg, q)];
                x[4 * q] = v.x;
                x[4 * q + 1] = v.y;
                x[4 * q + 2] = v.z;
                x[4 * q + 3] = v.w;
            }
        } else {
#pragma unroll
            for (int w = 0; w < N; w++) x[w] = a[seg * N + w];
        }
    }
    template <int N>
    static __device__ __forceinline__ void store(uint32_t* a, uint32_t seg, const uint32_t (&x)[N]) {
        if constexpr (M > 8) {
#pragma unroll
            for (int q = 0; q < N / 4; q++)
                reinterpret_cast<uint4*>(a)[word<N>(seg, q)] =
                    make_uint4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
        } else {
#pragma unroll
            for (int w = 0; w < N; w++) a[seg * N + w] = x[w];
        }
    }
};

template <int M, int THREADS>
constexpr size_t group_scratch_bytes() {
    return sizeof(GroupScratch<M, THREADS>);
}

// Class counts of one thread's elements, a byte per class (a thread owns at most
// 36): in registers up to 8 classes, in the thread's column above.
template <int M, int THREADS>
struct GroupCounts {
    using GS = GroupScratch<M, THREADS>;
    uint64_t w;
    unsigned char* mine;
    __device__ __forceinline__ void init(GS& gs) {
        w = 0;
        if constexpr (M > 8) {
            mine = reinterpret_cast<unsigned char*>(&gs.col[0][threadIdx.x]);
#pragma unroll
            for (int q = 0; q < GS::NB; q++) gs.col[q][threadIdx.x] = 0u;
        }
    }
    __device__ __forceinline__ void inc(uint32_t c) {
        if constexpr (M <= 4) {
            w = static_cast<uint32_t>(w) + (1u << (c << 3));
        } else if constexpr (M <= 8) {
            w += 1ull << (c << 3);
        } else {
            unsigned char& x = mine[(c >> 2) * (4u * THREADS) + (c & 3u)];
            x = static_cast<unsigned char>(x + 1u);
        }
    }
    __device__ __forceinline__ uint32_t word(const GS& gs, int q) const {
        if constexpr (M > 8) return gs.col[q][threadIdx.x];
        else return static_cast<uint32_t>(w >> (32 * q));
    }
};

// 16-bit pairs (classes 2 i, 2 i + 1) of a word of byte counts.
__device__ __forceinline__ uint32_t widen_lo(uint32_t x) { return __byte_perm(x, 0u, 0x4140); }
__device__ __forceinline__ uint32_t widen_hi(uint32_t x) { return __byte_perm(x, 0u, 0x4342); }
template <int M>
__device__ __forceinline__ uint32_t widen_pair(uint32_t x, int h) {  // pair h of word h / 2
    return (h & 1) ? widen_hi(x) : widen_lo(x);
}

// Where a thread's next element of each class goes: 16-bit fields, in registers up
// to 4 classes, in the thread's column above.
template <int M, int THREADS>
struct GroupCursors {
    using GS = GroupScratch<M, THREADS>;
    uint64_t w;
    unsigned char* mine;
    __device__ __forceinline__ void init(GS& gs) {
        mine = reinterpret_cast<unsigned char*>(&gs.col[0][threadIdx.x]);
        w = 0;
    }
    __device__ __forceinline__ void set(GS& gs, int h, uint32_t x) {
        if constexpr (M == 2) w = x;
        else if constexpr (M == 4) w = h == 0 ? ((w >> 32) << 32 | x) : ((w & 0xffffffffull) | static_cast<uint64_t>(x) << 32);
        else gs.col[h][threadIdx.x] = x;
    }
    __device__ __forceinline__ uint32_t next(uint32_t c) {
        if constexpr (M == 2) {
            const uint32_t x = static_cast<uint32_t>(w);
            w = x + (1u << (c << 4));
            return (x >> (c << 4)) & 0xffffu;
        } else if constexpr (M == 4) {
            const uint32_t p = static_cast<uint32_t>(w >> (c << 4)) & 0xffffu;
            w += 1ull << (c << 4);
            return p;
        } else {
            uint16_t& x = *reinterpret_cast<uint16_t*>(mine + (c >> 1) * (4u * THREADS) + (c & 1u) * 2u);
            const uint32_t p = x;
            x = static_cast<uint16_t>(p + 1u);
            return p;
        }
    }
};

// Offsets (and class count) of segment h + threadIdx.x of the next group,
// loaded by each thread while the current group is partitioned.
struct GroupPrefetch {
    uint64_t o0, o1;
    uint32_t m;
    bool valid;
};

// The discriminator of a group's segment with class count m: per-segment
// remainders use the precomputed constants cmod[m] (DiscrMod::make).
template <class D>
__device__ __forceinline__ D group_discr(const SegArgs& a, const D& d, const uint32_t* cmod,
                                         uint32_t m) {
    if constexpr (std::is_same<D, DiscrMod>::value) {
        if (a.seg_m != nullptr) {
            DiscrMod x;
            x.m = min(m, 16u);
            x.c = cmod[x.m];
            return x;
        }
    }
    return d;
}

// One CTA partitions one group of small segments held in shared memory (its element
// y at src[y], phase <= y < end) into the output image dst and writes the segments'
// sizes.  Every thread owns k consecutive positions whatever the segment lengths, k
// an odd number of 16-byte words (a warp's loads then fall in different banks):
//   heads   one thread per segment publishes its head; each thread finds the first
//           head at or after its own range (binary search);
//   counts  class counts of the thread's elements; where a head lies inside, the
//           counts so far are noted for it.  A 16-byte word without a head in it
//           (all but one in a thousand for segments of a thousand) takes no test;
//   scan    exclusive 16-bit class counts over the threads, segments disregarded;
//   sizes   one thread per segment: the group's class counts before its head and
//           before the next give its sizes, and with them where each class begins;
//   place   every element to the next position of its class: at a head those of the
//           segment, before it those of the segment the thread's range begins in
//           (its first positions plus what lies between its head and the range).
// The counts are kept per class and never per segment, so no scan carries segment
// flags and no thread closes a segment for the others.  6 * 10^7 u32 in segments
// of up to 4096 (mean 1600), m = 4: 46 instructions an element and 167 us, where a
// segmented scan with the segments closed by the threads that hold their ends took
// 78 and 212; 10^5 LogNormal(ln 1024, 1.5) segments, m = 4, 8, 16: 368, 457, 745 ->
// 306, 361, 689 us, with the groups' ranges fetched ahead (GroupRange) 289, 349, 633.  What bounds it now is latency: four barriers
// a group and 24 warps to an SM (shared memory).  Windows of P / 2 with
// four CTAs: 299 against 289 us at m = 4, 439 against 349 at m = 8, 663 against 633
// at m = 16; windows of 3 P / 4 were slower too.  The run counts as items of this kernel, to fill the idle memory
// pipe: 545 us for both against 306 + 157.
template <class V, class D, int M, int THREADS>
__device__ __forceinline__ void seg_group_cta(const SegArgs& a, const D& d, const uint32_t* cmod,
                                              uint32_t h, uint32_t nseg, uint64_t as, uint32_t phase,
                                              uint32_t end, const V* src, V* dst,
                                              GroupScratch<M, THREADS>& gs, uint32_t qn0, uint32_t nq) {
    using GS = GroupScratch<M, THREADS>;
    constexpr int NB = GS::NB, NH = GS::NH;
    constexpr int W = THREADS / 32;
    constexpr uint32_t VE = 16 / sizeof(V);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t k = nq * VE, lo = static_cast<uint32_t>(tid) * k;

    // ---- counts
    GroupCounts<M, THREADS> cnt;
    cnt.init(gs);
    {
        uint32_t qn = qn0, nxt = gs.hpos[qn0];
        D dc = group_discr(a, d, cmod, qn > 0u ? gs.msz[qn - 1u] : a.m);
        for (uint32_t j = 0; j < nq; j++) {
            const uint32_t y0 = lo + j * VE;
            if (y0 >= end) break;
            V v[VE];
            unpack16_to<V>(*reinterpret_cast<const uint4*>(src + y0), v);
            if (nxt >= y0 + VE) {
#pragma unroll
                for (uint32_t e = 0; e < VE; e++) cnt.inc(dc(v[e]));
            } else {
#pragma unroll
                for (uint32_t e = 0; e < VE; e++) {
                    const uint32_t y = y0 + e;
                    while (nxt == y && qn < nseg) {
                        uint32_t own[NB];
#pragma unroll
                        for (int q = 0; q < NB; q++) own[q] = cnt.word(gs, q);
                        GS::store(gs.hcnt, qn, own);
                        dc = group_discr(a, d, cmod, gs.msz[qn]);
                        nxt = gs.hpos[++qn];
                    }
                    if (qn > 0u && y < end) cnt.inc(dc(v[e]));
                }
            }
        }
    }

    // ---- scan over the threads: exclusive counts within the warp, warp totals
    uint32_t inc[NH];
    {
        uint32_t own[NH];
#pragma unroll
        for (int i = 0; i < NH; i++) own[i] = widen_pair<M>(cnt.word(gs, i / 2), i);
#pragma unroll
        for (int i = 0; i < NH; i++) {
            inc[i] = warp_incl_scan(own[i]);
            if (lane == 31) gs.wagg[i][warp] = inc[i];
            inc[i] -= own[i];
            gs.col[i][tid] = inc[i];
        }
    }
    __syncthreads();
    // the warps before this one, by the first lanes of every warp (lane w: warp w)
    uint32_t wpre[NH], tot[NH];  // lane w: counts before warp w; the group's
#pragma unroll
    for (int i = 0; i < NH; i++) {
        const uint32_t x = lane < W ? gs.wagg[i][lane] : 0u;
        uint32_t in = x;
#pragma unroll
        for (int dd = 1; dd < W; dd <<= 1) {
            const uint32_t up = __shfl_up_sync(0xffffffffu, in, dd);
            if (lane >= dd) in += up;
        }
        wpre[i] = in - x;
        tot[i] = __shfl_sync(0xffffffffu, in, W - 1);
        inc[i] += __shfl_sync(0xffffffffu, wpre[i], warp);
    }

    // ---- sizes (whole warps, so that the warp totals can be looked up by shuffles)
    if (static_cast<uint32_t>(warp) * 32u < nseg) {
        const bool mine = static_cast<uint32_t>(tid) < nseg;
        const uint32_t hq = gs.hpos[mine ? tid : 0], hn = gs.hpos[mine ? tid + 1 : 0];
        uint32_t p0[NH], p1[NH];
        auto before = [&](uint32_t q, uint32_t y, uint32_t (&p)[NH]) {  // counts before head q at y
            const bool inside = y < end && q < nseg;
            const uint32_t t = inside ? y / k : 0u;
            uint32_t own[NB];
            GS::load(gs.hcnt, inside ? q : 0u, own);
#pragma unroll
            for (int i = 0; i < NH; i++) {
                const uint32_t w = __shfl_sync(0xffffffffu, wpre[i], t >> 5);
                p[i] = inside ? w + gs.col[i][t] + widen_pair<M>(own[i / 2], i) : tot[i];
            }
        };
        before(tid, hq, p0);
        before(tid + 1, hn, p1);
        const uint64_t s = static_cast<uint64_t>(h) + tid;
        uint32_t off = 0;
        if (mine) {
            uint32_t cur[NH];
#pragma unroll
            for (int i = 0; i < NH; i++) {
                const uint32_t n = p1[i] - p0[i];  // each 16-bit field is no smaller
                const uint32_t n0 = n & 0xffffu, n1 = n >> 16;
                const uint32_t o0 = off, o1 = off + n0;
                off = o1 + n1;
                cur[i] = (hq + o0) | ((hq + o1) << 16);
                if (a.seg_sizes != nullptr) {
                    if (2u * i < a.m) a.seg_sizes[s * a.m + 2 * i] = n0;
                    if (2u * i + 1u < a.m) a.seg_sizes[s * a.m + 2 * i + 1] = n1;
                }
                if (a.headflags != nullptr) {
                    if (n0 > 0u) a.headflags[as + hq + o0] = n0;
                    if (n1 > 0u) a.headflags[as + hq + o1] = n1;
                }
            }
            GS::store(gs.hpre, tid, p0);
            GS::store(gs.hcur, tid, cur);
        }
    }
    // the output image is about to be rewritten: the previous group's bulk store
    // must have finished reading it
    if (tid == 0) bulk_wait_read<0>();
    __syncthreads();

    // ---- place
    {
        uint32_t qn = qn0, nxt = gs.hpos[qn0];
        D dc = group_discr(a, d, cmod, qn > 0u ? gs.msz[qn - 1u] : a.m);
        GroupCursors<M, THREADS> cur;
        cur.init(gs);
        if (qn > 0u) {
            uint32_t first[NH], before[NH];
            GS::load(gs.hcur, qn - 1u, first);
            GS::load(gs.hpre, qn - 1u, before);
#pragma unroll
            for (int i = 0; i < NH; i++) cur.set(gs, i, first[i] + (inc[i] - before[i]));
        }
        for (uint32_t j = 0; j < nq; j++) {
            const uint32_t y0 = lo + j * VE;
            if (y0 >= end) break;
            V v[VE];
            unpack16_to<V>(*reinterpret_cast<const uint4*>(src + y0), v);
            if (nxt >= y0 + VE) {
#pragma unroll
                for (uint32_t e = 0; e < VE; e++) dst[cur.next(dc(v[e]))] = v[e];
            } else {
#pragma unroll
                for (uint32_t e = 0; e < VE; e++) {
                    const uint32_t y = y0 + e;
                    while (nxt == y && qn < nseg) {
                        uint32_t first[NH];
                        GS::load(gs.hcur, qn, first);
#pragma unroll
                        for (int i = 0; i < NH; i++) cur.set(gs, i, first[i]);
                        dc = group_discr(a, d, cmod, gs.msz[qn]);
                        nxt = gs.hpos[++qn];
                    }
                    if (qn > 0u && y < end) dst[cur.next(dc(v[e]))] = v[e];
                }
            }
        }
    }
}

// The class counts of run j of a large segment by one CTA: 16-byte loads eight deep
// per thread, per-thread packed counters, warp reductions and one barrier (`red` is
// used in turns by the caller's parity).
template <class V, class D, int M, int THREADS>
__device__ __forceinline__ void count_run(const SegArgs& a, const D& d, uint32_t j,
                                          uint32_t (*red)[M]) {
    constexpr uint32_t AU = 16 / sizeof(V);
    constexpr int W = THREADS / 32;
    constexpr int UNROLL = M <= 8 ? 8 : 4;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const V* in = static_cast<const V*>(a.in);
    const bool in_vec = (reinterpret_cast<uintptr_t>(in) & 15u) == 0;
    const RunEntry ent = a.runs[j];
    const D dj = seg_discr(a, d, ent.len_m >> 24);
    PackedCounts<M> pc;
    pc.init();
    const uint64_t p0 = ent.p0, p1 = ent.p1();
    const uint64_t vs = in_vec ? min((p0 + AU - 1u) & ~static_cast<uint64_t>(AU - 1u), p1) : p1;
    const uint64_t ve = in_vec ? max(vs, p1 & ~static_cast<uint64_t>(AU - 1u)) : p1;
    uint32_t k = 0;
    auto edge = [&](uint64_t e) {
        pc.add(dj(in[e]));
        if (++k == 8u) {
            pc.fold();
            k = 0;
        }
    };
    for (uint64_t e = p0 + tid; e < vs; e += THREADS) edge(e);
    for (uint64_t e = ve + tid; e < p1; e += THREADS) edge(e);
    pc.fold();
    const uint4* vp = reinterpret_cast<const uint4*>(in + vs);
    const uint32_t nv = static_cast<uint32_t>((ve - vs) / AU);
    for (uint32_t q = tid; q < nv; q += THREADS * UNROLL) {
        uint4 r[UNROLL];
#pragma unroll
        for (int uu = 0; uu < UNROLL; uu++)
            if (q + uu * THREADS < nv) r[uu] = __ldg(vp + q + uu * THREADS);
#pragma unroll
        for (int uu = 0; uu < UNROLL; uu++) {
            if (q + uu * THREADS < nv) {
                V e[AU];
                unpack16_to<V>(r[uu], e);
#pragma unroll
                for (uint32_t z = 0; z < AU; z++) pc.add(dj(e[z]));
            }
            if (uu & 1) pc.fold();  // every two vectors: <= 8 increments
        }
    }
    pc.finish();
#pragma unroll
    for (int c = 0; c < M; c++) {
        const uint32_t x = warp_sum(pc.acc[c]);
        if (lane == 0) red[warp][c] = x;
    }
    __syncthreads();
    if (tid < static_cast<uint32_t>(M)) {
        uint32_t agg = 0;
#pragma unroll
        for (int w = 0; w < W; w++) agg += red[w][tid];
        a.run_cnt[static_cast<uint64_t>(j) * M + tid] = agg;
    }
}

// The class counts of every run of the large segments, one CTA per run.
template <class V, class D, int M, int THREADS>
__global__ void __launch_bounds__(THREADS, 4) seg_run_count(SegArgs a, D d) {
    __shared__ uint32_t red[2][THREADS / 32][M];
    __shared__ uint32_t ticket_sh[2];
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t num_runs = a.hdr->num_runs;
    for (uint32_t it = 0;; it++) {
        if (threadIdx.x == 0) ticket_sh[it & 1u] = atomicAdd(&a.hdr->ticket3, 1u);
        __syncthreads();
        const uint32_t j = ticket_sh[it & 1u];
        if (j >= num_runs) break;
        count_run<V, D, M, THREADS>(a, d, j, red[it & 1u]);
    }
}

// A CTA's groups in their pipeline: a group's ticket is drawn four groups ahead, its
// entry loaded three, its range loaded two and published one group ahead, all by one
// thread of the last warp, so that no group waits for that chain.  Loaded at a
// batch's start, the chain and its two barriers were 306 against 289 us on 10^5
// LogNormal(ln 1024, 1.5) segments (u32, m = 4, batches of two groups; in batches of
// sixteen, which hid it before, 314: their last ones leave CTAs idle).  Without
// tickets, the groups dealt out in turns: 307.
struct GroupRange {
    uint32_t h, he;   // segments [h, he)
    uint32_t r0, r1;  // elements [r0, r1) (n < 2^32)
    uint32_t valid;   // false: the CTA has had its last group
};

// Persistent; CTA b begins with batch b of the small-segment groups and takes tickets
// for the batches after its first.
template <class V, class D, int M, int THREADS>
__global__ void __launch_bounds__(THREADS, 3)
    seg_main(SegArgs a, D d) {
    using L = SegSmem<V, M, THREADS>;
    constexpr uint32_t AU = L::kAU;
    constexpr uint32_t P = L::kTile;
    constexpr int kPlanner = THREADS - 1;  // the thread that knows the groups to come
    static_assert(M <= 16 && M >= 2, "class bound");
    static_assert(static_cast<int>(kGroupSegs) <= THREADS, "one thread per segment");
    static_assert(3 * (L::kBytes + L::kReserved) <= L::kSmBytes, "three CTAs to an SM");

    extern __shared__ __align__(128) unsigned char smem_raw[];
    const uint32_t raw = smem_addr(smem_raw);
    unsigned char* base = smem_raw + (((raw + 127u) & ~127u) - raw);
    V* g_in = reinterpret_cast<V*>(base);
    V* g_out = g_in + L::kGroupElems;
    GroupScratch<M, THREADS>& gs = *reinterpret_cast<GroupScratch<M, THREADS>*>(g_out + L::kGroupElems);

    __shared__ __align__(8) uint64_t gbar;
    __shared__ GroupRange range_sh[2];  // of this group and of the next, in turns
    __shared__ uint32_t cmod[17];  // DiscrMod constants for m = 1 .. 16

    const int tid = threadIdx.x;
    const V* in = static_cast<const V*>(a.in);
    V* out = static_cast<V*>(a.out);
    const bool in_vec = (reinterpret_cast<uintptr_t>(in) & 15u) == 0;
    const bool out_vec = (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
    pdl_launch_dependents();
    pdl_wait();
    const uint64_t S = seg_count(a);
    const uint32_t num_groups = a.hdr->num_groups;
    // neighbouring groups per ticket: the tuned batch, but no more than spreads the
    // groups over every CTA (a few groups must not queue up on one CTA)
    const uint32_t batch =
        max(1u, min(a.group_batch, (num_groups + gridDim.x - 1) / gridDim.x));
    uint32_t uses = 0;  // of the input buffer

    // kPlanner's state: the group to load an entry of, `left` more of its batch, the
    // ticket after it; the entry; and of the group before that segments and elements
    uint32_t g = blockIdx.x * batch, left = batch - 1u, ticket = 0;
    uint32_t eh = 0, ee = 0, wh = 0, we = 0;
    bool ev = false, wv = false, cut = false;  // cut: what is left is the group's last segment
    uint64_t w0 = 0, w1 = 0, wl = 0;           // its elements; where its last segment begins
    constexpr uint32_t kMost = L::kGroupMost;
    constexpr bool kCut = kMost < 2u * P;
    auto draw = [&] { ticket = gridDim.x + atomicAdd(&a.hdr->ticket, 1u); };
    auto load_entry = [&] {  // of group g, then the next group
        ev = g < num_groups;
        if (!ev) return;
        eh = a.groups[g];
        ee = a.groups_end[g];
        g++;
        if (left-- == 0u) {
            g = ticket * batch;
            left = batch - 1u;
            draw();
        }
    };
    auto load_range = [&] {  // of the entry
        wv = ev;
        if (!ev) return;
        wh = eh;
        we = static_cast<uint32_t>(min(static_cast<uint64_t>(ee), S));
        we = min(max(we, wh), wh + kGroupSegs);
        w0 = a.offsets[wh];
        w1 = a.offsets[we];
        if constexpr (kCut) wl = a.offsets[max(we, 1u) - 1u];
    };
    auto publish = [&](uint32_t q) {  // true: the group's last segment is still to come
        cut = kCut && !cut && wv && w1 - w0 > kMost && w1 - w0 < 2u * P && we - wh > 1u;
        const uint64_t end = cut ? wl : w1;
        const bool bad = end < w0 || end - w0 > kMost || end > a.n;  // malformed: nothing to do
        range_sh[q].h = wh;
        range_sh[q].he = bad ? wh : cut ? we - 1u : we;
        range_sh[q].r0 = bad ? 0u : static_cast<uint32_t>(w0);
        range_sh[q].r1 = bad ? 0u : static_cast<uint32_t>(end);
        range_sh[q].valid = wv;
        if (cut) {
            wh = we - 1u;
            w0 = wl;
        }
        return cut;
    };
    auto fetch = [&] {
        load_range();
        load_entry();
    };
    // the 16-byte words of a group that one bulk copy brings
    auto vec_end = [&](uint32_t r1, uint64_t as) {
        const uint64_t ve = min((static_cast<uint64_t>(r1) + AU - 1u) & ~static_cast<uint64_t>(AU - 1u),
                                a.n & ~static_cast<uint64_t>(AU - 1u));
        return in_vec && ve > as ? ve : as;
    };
    auto issue_group = [&](uint32_t q) {  // thread 0 only
        const uint64_t as = range_sh[q].r0 & ~(AU - 1u);
        const uint32_t bytes = static_cast<uint32_t>((vec_end(range_sh[q].r1, as) - as) * sizeof(V));
        if (bytes > 0) {
            mbar_arrive_expect_tx(&gbar, bytes);
            bulk_load_g2s(g_in, in + as, bytes, &gbar);
        } else {
            mbar_arrive(&gbar);
        }
    };

    if (tid == 0) {
        mbar_init(&gbar, 1);
        mbar_fence_init();
    }
    if (tid >= 1 && tid <= 16) cmod[tid] = DiscrMod::make(static_cast<uint32_t>(tid)).c;
    if (tid == 0) cmod[0] = 0;
    if (g >= num_groups) return;
    if (tid == kPlanner) {
        draw();
        load_entry();
        load_range();
        load_entry();
        if (!publish(0)) fetch();
    }
    __syncthreads();
    if (tid == 0) issue_group(0);

    GroupPrefetch pf;
    pf.valid = false;
    for (uint32_t q = 0; range_sh[q].valid; q ^= 1u) {
        const uint32_t h = range_sh[q].h, nseg = range_sh[q].he - h;
        const uint32_t r0 = range_sh[q].r0, r1 = range_sh[q].r1;
        if (tid == kPlanner) {
            if (!publish(q ^ 1u)) fetch();
        }
        const uint64_t as = r0 & ~static_cast<uint64_t>(AU - 1u);
        const uint32_t phase = static_cast<uint32_t>(r0 - as);
        const uint32_t end = static_cast<uint32_t>(r1 - as);
        // ---- heads, while the group's elements are on their way
        bool bad = false;
        if (static_cast<uint32_t>(tid) < nseg) {
            if (!pf.valid) {
                pf.o0 = a.offsets[h + tid];
                pf.o1 = a.offsets[h + tid + 1];
                pf.m = a.seg_m != nullptr ? min(max(a.seg_m[h + tid], 1u), a.m_bound) : a.m;
            }
            bad = pf.o0 < r0 || pf.o1 < pf.o0 || pf.o1 > r1;
            gs.hpos[tid] = static_cast<uint16_t>(pf.o0 - as);
            gs.msz[tid] = static_cast<uint8_t>(pf.m);
        }
        if (tid == 0) gs.hpos[nseg] = static_cast<uint16_t>(end);
        const bool ok = mbar_wait_bounded(&gbar, uses & 1u);
        const uint64_t ve = vec_end(r1, as);
        if (ve < r1) {  // what the bulk copy did not bring (CTA-uniform)
            for (uint64_t e = max(ve, static_cast<uint64_t>(r0)) + tid; e < r1; e += THREADS)
                g_in[e - as] = in[e];
        }
        if (__syncthreads_or(bad || !ok)) {  // a malformed group is left alone
            fence_proxy_async_smem();
            if (__syncthreads_or(!ok)) {
                if (tid == 0) {  // only this group's copy can be in flight
                    const bool late = mbar_wait_bounded(&gbar, uses & 1u);
                    if (!late) atomicOr(&a.hdr->error, kErrTimeout);
                }
                break;
            }
            uses++;
            pf.valid = false;
            if (tid == 0 && range_sh[q ^ 1u].valid) issue_group(q ^ 1u);
            continue;
        }
        uses++;
        const bool more = range_sh[q ^ 1u].valid;
        pf.valid = more;
        if (more && static_cast<uint32_t>(tid) < range_sh[q ^ 1u].he - range_sh[q ^ 1u].h) {
            const uint64_t ns = static_cast<uint64_t>(range_sh[q ^ 1u].h) + tid;
            pf.o0 = a.offsets[ns];
            pf.o1 = a.offsets[ns + 1];
            pf.m = a.seg_m != nullptr ? min(max(a.seg_m[ns], 1u), a.m_bound) : a.m;
        }
        const uint32_t nq = ((end + THREADS * AU - 1u) / (THREADS * AU)) | 1u;
        uint32_t qn = 0;  // heads before the thread's first position
        if (nseg > 0u) {
            const uint32_t lo = static_cast<uint32_t>(tid) * nq * AU;
            for (uint32_t step = 1u << (31 - __clz(nseg)); step > 0u; step >>= 1)
                if (qn + step <= nseg && gs.hpos[qn + step - 1u] < lo) qn += step;
        }
        seg_group_cta<V, D, M, THREADS>(a, d, cmod, h, nseg, as, phase, end, g_in, g_out, gs, qn, nq);
        // every access of the buffers precedes the copies of them
        fence_proxy_async_smem();
        __syncthreads();
        if (tid == 0 && more) issue_group(q ^ 1u);
        // write the range back from the output image
        const uint32_t vs = min((phase + AU - 1u) & ~(AU - 1u), end), vt = max(vs, end & ~(AU - 1u));
        if (out_vec) {
            if (tid == 0 && vt > vs) {
                bulk_store_s2g(out + as + vs, g_out + vs, (vt - vs) * sizeof(V));
                bulk_commit();
            }
            if (static_cast<uint32_t>(tid) < vs - phase) out[r0 + tid] = g_out[phase + tid];
            if (static_cast<uint32_t>(tid) < end - vt) out[as + vt + tid] = g_out[vt + tid];
        } else {
            for (uint32_t y = phase + tid; y < end; y += THREADS) out[as + y] = g_out[y];
            __syncthreads();
        }
    }
    if (tid == 0) bulk_wait_all();
}

// A row of M u32 words in 16-byte (8-byte) accesses.
template <int M>
__device__ __forceinline__ void load_row(const uint32_t* p, uint32_t (&x)[M]) {
    if constexpr (M == 2) {
        const uint2 v = __ldcg(reinterpret_cast<const uint2*>(p));
        x[0] = v.x;
        x[1] = v.y;
    } else {
#pragma unroll
        for (int q = 0; q < M / 4; q++) {
            const uint4 v = __ldcg(reinterpret_cast<const uint4*>(p) + q);
            x[4 * q] = v.x;
            x[4 * q + 1] = v.y;
            x[4 * q + 2] = v.z;
            x[4 * q + 3] = v.w;
        }
    }
}
template <int M>
__device__ __forceinline__ void store_row(uint32_t* p, const uint32_t (&x)[M]) {
    if constexpr (M == 2) {
        *reinterpret_cast<uint2*>(p) = make_uint2(x[0], x[1]);
    } else {
#pragma unroll
        for (int q = 0; q < M / 4; q++)
            reinterpret_cast<uint4*>(p)[q] = make_uint4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
    }
}

// One large segment's runs [j, jl]: lane l takes a contiguous share of the
// runs, class counts in registers; warp scans per class give each run's
// output position per class, the segment's sizes and head flags.  A lane has
// several rows in flight: a segment of many runs is one chain of loads otherwise
// (one segment of 3 * 10^7 8-byte records, m = 2, 7325 runs: 242 us a call with one row
// in flight, 173 with eight).
template <int M>
__device__ __forceinline__ void scan_segment_runs(const SegArgs& a, uint32_t j, uint32_t jl,
                                                  uint32_t seg, uint32_t seg_start) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t R = jl - j + 1u;
    const uint32_t per = (R + 31u) >> 5;
    const uint32_t rb = j + min(lane * per, R), re = j + min(lane * per + per, R);
    constexpr uint32_t U = M <= 4 ? 8 : 4;
    uint32_t acc[M], x[U][M];
    auto load = [&](uint32_t r) {
#pragma unroll
        for (uint32_t u = 0; u < U; u++) {
            if (r + u < re) {
                load_row<M>(a.run_cnt + static_cast<uint64_t>(r + u) * M, x[u]);
            } else {
#pragma unroll
                for (int c = 0; c < M; c++) x[u][c] = 0u;
            }
        }
    };
#pragma unroll
    for (int c = 0; c < M; c++) acc[c] = 0;
    for (uint32_t r = rb; r < re; r += U) {
        load(r);
#pragma unroll
        for (uint32_t u = 0; u < U; u++)
#pragma unroll
            for (int c = 0; c < M; c++) acc[c] += x[u][c];
    }
    uint32_t cur[M];
    uint32_t off = seg_start;
#pragma unroll
    for (int c = 0; c < M; c++) {
        const uint32_t incl = warp_incl_scan(acc[c]);
        const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
        cur[c] = off + incl - acc[c];
        if (lane == static_cast<uint32_t>(c)) {
            if (a.seg_sizes != nullptr && static_cast<uint32_t>(c) < a.m)
                a.seg_sizes[static_cast<uint64_t>(seg) * a.m + c] = tot;
            if (a.headflags != nullptr && tot > 0) a.headflags[off] = tot;
        }
        off += tot;
    }
    for (uint32_t r = rb; r < re; r += U) {
        if (per > U) load(r);
#pragma unroll
        for (uint32_t u = 0; u < U; u++) {
            if (r + u < re) store_row<M>(a.run_base + static_cast<uint64_t>(r + u) * M, cur);
#pragma unroll
            for (int c = 0; c < M; c++) cur[c] += x[u][c];
        }
    }
}

// One large segment with at most kLaneRuns runs [j, jl], by one lane alone, the
// counts of all of them in flight at once.
constexpr uint32_t kLaneRuns = 4;
template <int M>
__device__ __forceinline__ void scan_segment_runs_lane(const SegArgs& a, uint32_t j, uint32_t jl,
                                                       uint32_t seg, uint32_t seg_start) {
    uint32_t x[kLaneRuns][M], cur[M];
#pragma unroll
    for (uint32_t r = 0; r < kLaneRuns; r++) {
        if (j + r <= jl) {
            load_row<M>(a.run_cnt + static_cast<uint64_t>(j + r) * M, x[r]);
        } else {
#pragma unroll
            for (int c = 0; c < M; c++) x[r][c] = 0u;
        }
    }
    uint32_t off = seg_start;
#pragma unroll
    for (int c = 0; c < M; c++) {
        uint32_t tot = 0;
#pragma unroll
        for (uint32_t r = 0; r < kLaneRuns; r++) tot += x[r][c];
        cur[c] = off;
        if (a.seg_sizes != nullptr && static_cast<uint32_t>(c) < a.m)
            a.seg_sizes[static_cast<uint64_t>(seg) * a.m + c] = tot;
        if (a.headflags != nullptr && tot > 0) a.headflags[off] = tot;
        off += tot;
    }
#pragma unroll
    for (uint32_t r = 0; r < kLaneRuns; r++) {
        if (j + r <= jl) store_row<M>(a.run_base + static_cast<uint64_t>(j + r) * M, cur);
#pragma unroll
        for (int c = 0; c < M; c++) cur[c] += x[r][c];
    }
}

// Every warp looks at up to 32 consecutive runs at a time (fewer when there are few:
// the long segments in a warp's part are scanned one after the other): the lane
// holding a segment's first run scans a segment of at most kLaneRuns runs by itself,
// the whole warp takes the longer ones in turn.
template <int M>
__global__ void __launch_bounds__(256) seg_run_scan(SegArgs a) {
    const uint32_t lane = threadIdx.x & 31u;
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t num_runs = a.hdr->num_runs;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t per = min(32u, (num_runs + warps - 1u) / warps);
    for (uint32_t j0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * per; j0 < num_runs;
         j0 += warps * per) {
        const uint32_t j = j0 + lane;
        RunEntry e{};
        bool first = false;
        if (lane < per && j < num_runs) {
            e = a.runs[j];
            first = j == 0u || a.runs[j - 1u].seg != e.seg;
        }
        const uint32_t jl = min(e.jlast, num_runs - 1u);
        const bool shortseg = first && jl >= j && jl - j < kLaneRuns;
        if (shortseg) scan_segment_runs_lane<M>(a, j, jl, e.seg, e.p0);
        uint32_t longs = __ballot_sync(0xffffffffu, first && !shortseg);
        while (longs != 0u) {
            const int l = __ffs(longs) - 1;
            longs &= longs - 1u;
            const uint32_t jll = __shfl_sync(0xffffffffu, jl, l);
            const uint32_t seg = __shfl_sync(0xffffffffu, e.seg, l);
            const uint32_t p0 = __shfl_sync(0xffffffffu, e.p0, l);
            if (jll >= j0 + l) scan_segment_runs<M>(a, j0 + l, jll, seg, p0);
        }
    }
}

// Every run of a large segment through a TMA slot and the tile step, from the
// run_base positions.  Runs are taken in reverse order of the counts, so
// the first re-reads find the runs counted last still in L2.
//
// A run is 2.5 tiles on average, so what it needs before its first tile is fetched
// during the run before: its ticket is drawn at the last tile of the run before
// that, its entry is loaded (by one thread of the last warp, which waits for nothing
// it has not had a tile's time for) while that run is placed, and at that run's last
// tile its first tile and its class positions are requested.
template <class V, class D, int M, int THREADS>
__global__ void __launch_bounds__(THREADS, 4)  // 4 CTAs (32 warps) per SM: <= 64 registers
    seg_run_scatter(SegArgs a, D d, const __grid_constant__ CUtensorMap tmap) {
    using L = RunSmem<V, M, THREADS>;
    using TG = typename L::G;
    constexpr int ITEMS = TG::kItems;
    constexpr int P = TG::kTile;
    constexpr int ROWS = TG::kRows;
    constexpr uint32_t AU = TG::kAU;
    static_assert(M <= 16 && M >= 2, "class bound");
    static_assert(ROWS <= 256, "TMA box height");

    extern __shared__ __align__(128) unsigned char smem_raw[];
    const uint32_t raw = smem_addr(smem_raw);
    unsigned char* base = smem_raw + (((raw + 1023u) & ~1023u) - raw);
    V* slot = reinterpret_cast<V*>(base);
    V* stage = reinterpret_cast<V*>(base + L::kSlotBytes);
    uint32_t* cnt_sm = reinterpret_cast<uint32_t*>(base + L::kSlotBytes + TG::kStageBytes);

    __shared__ __align__(8) uint64_t bar;
    __shared__ TileShared<M> sh;
    __shared__ RunEntry ent_sh[2];  // by parity of the run
    __shared__ uint32_t run_sh[2];  // its index, or kNoRun

    constexpr uint32_t kNoRun = 0xffffffffu;
    constexpr int kFetcher = THREADS - 32;
    const int tid = threadIdx.x;
    const V* in = static_cast<const V*>(a.in);
    V* out = static_cast<V*>(a.out);
    const uint32_t out_phase =
        static_cast<uint32_t>(reinterpret_cast<uintptr_t>(out) / sizeof(V)) & (AU - 1u);
    const bool tma_ok = a.use_tma != 0;
    constexpr uint32_t kPerRow = 128u / sizeof(V);  // elements per 128-byte row
    const uint64_t map_elems = (a.n * sizeof(V) / 128u) * kPerRow;
    if (tid == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
    }
    pdl_wait();
    const uint32_t num_runs = a.hdr->num_runs;

    // the run's tiles start at the 128-byte row holding its first element
    // (not at multiples of P), so only its last tile is short
    auto row_start = [&](const RunEntry& e) {
        return static_cast<uint64_t>(e.p0 & ~(kPerRow - 1u));
    };
    // a tile comes by TMA when the run's part of it lies inside the tensor
    // map (the input's whole 128-byte rows; rows past the map read as zeros
    // and lie outside the run)
    auto via_tma = [&](const RunEntry& e, uint32_t i) {
        return tma_ok && min(static_cast<uint64_t>(e.p1()),
                             row_start(e) + static_cast<uint64_t>(i + 1) * P) <= map_elems;
    };
    auto issue = [&](const RunEntry& e, uint32_t i) {  // thread 0: tile i of a run
        if (via_tma(e, i)) {
            mbar_arrive_expect_tx(&bar, P * sizeof(V));
            tma_load_2d(slot, &tmap, 0,
                        static_cast<int32_t>(row_start(e) / kPerRow + static_cast<uint64_t>(i) * ROWS),
                        &bar);
        } else {
            mbar_arrive(&bar);
        }
    };
    // kFetcher's state: the ticket of the run after the next known one, and its entry
    uint32_t ticket = 0;
    RunEntry next_ent{};
    bool have_next = false;
    auto fetch_entry = [&] {  // the entry of `ticket`'s run, used only later
        have_next = ticket < num_runs;
        if (have_next) next_ent = a.runs[num_runs - 1u - ticket];
    };
    auto publish = [&](uint32_t q) {
        ent_sh[q] = next_ent;
        run_sh[q] = have_next ? num_runs - 1u - ticket : kNoRun;
    };
    if (tid == kFetcher) {
        ticket = atomicAdd(&a.hdr->ticket2, 1u);
        fetch_entry();
        publish(0);
        ticket = have_next ? atomicAdd(&a.hdr->ticket2, 1u) : num_runs;
    }
    __syncthreads();
    if (run_sh[0] != kNoRun) {
        if (tid == 0) issue(ent_sh[0], 0);
        if (tid < M) sh.cursor[0][tid] = __ldcg(a.run_base + static_cast<uint64_t>(run_sh[0]) * M + tid);
    }

    const uint32_t e0 = tid * ITEMS;
    uint32_t uses = 0;  // of the slot
    bool failed = false;
    for (uint32_t q = 0; !failed && run_sh[q] != kNoRun; q ^= 1u) {
        const RunEntry ent = ent_sh[q];
        const D dj = seg_discr(a, d, ent.len_m >> 24);
        if (tid == kFetcher) fetch_entry();
        const uint64_t rb = row_start(ent);
        const uint32_t ntiles = static_cast<uint32_t>((ent.p1() - rb + P - 1u) / P);
        uint32_t next_cur = 0;
        for (uint32_t i = 0; i < ntiles; i++) {
            const uint64_t ts = rb + static_cast<uint64_t>(i) * P;
            const uint32_t lo = static_cast<uint32_t>(max(static_cast<uint64_t>(ent.p0), ts) - ts);
            const uint32_t hi = static_cast<uint32_t>(min(static_cast<uint64_t>(ent.p1()), ts + P) - ts);
            const bool full = lo == 0u && hi == static_cast<uint32_t>(P);
            const bool last = i + 1u == ntiles;
            const bool ok = mbar_wait_bounded(&bar, uses & 1u);
            V v[ITEMS];
            if (via_tma(ent, i)) {
                take_swizzled<V, ITEMS>(slot, v);
            } else {
#pragma unroll
                for (int z = 0; z < ITEMS; z++)
                    v[z] = (e0 + z >= lo && e0 + z < hi) ? in[ts + e0 + z] : V();
            }
            if (last && tid == kFetcher) {
                publish(q ^ 1u);
                ticket = have_next ? atomicAdd(&a.hdr->ticket2, 1u) : num_runs;
            }
            auto refill = [&] {  // the slot is free: the next tile of this run or of the next
                if (!last) {
                    if (tid == 0) issue(ent, i + 1u);
                } else if (run_sh[q ^ 1u] != kNoRun) {
                    if (tid == 0) issue(ent_sh[q ^ 1u], 0);
                    if (tid < M)
                        next_cur = __ldcg(a.run_base + static_cast<uint64_t>(run_sh[q ^ 1u]) * M + tid);
                }
            };
            bool done;
            if constexpr (M == 2)
                done = tile_filter<V, D, THREADS, true>(dj, v, lo, hi, full, stage, cnt_sm, sh, i & 1u,
                                                        OutFlat<V>{out, out_phase}, ok, refill);
            else
                done = tile_scatter<V, D, M, THREADS, true, false>(dj, v, lo, hi, full, stage, cnt_sm, sh,
                                                                   i & 1u, OutFlat<V>{out, out_phase},
                                                                   ok, refill);
            if (!done) {
                failed = true;
                if (tid == 0) {  // only this tile's copy can be in flight
                    atomicOr(&a.hdr->error, kErrTimeout);
                    (void)mbar_wait_bounded(&bar, uses & 1u);
                }
                break;
            }
            uses++;
        }
        // read after the next tile's first barrier; this run's last reads of the
        // cursors lie before its last tile's third
        if (tid < M) sh.cursor[0][tid] = next_cur;
    }
    if (tid < M) bulk_wait_all();
}

// ------------------------------------------------------- medium segments --
// A medium segment (more than one tile, at most mid_tiles <= KMAX row-aligned
// tiles) is read from HBM once: all its tiles come by TMA into a shared slab;
// a count pass over the slab gives the segment's class totals (its sizes, head
// flags and the class cursors at its start); tile_scatter then places the
// tiles from the slab in order with forward cursors, as the plain scatter
// does.  The run path reads the same elements twice (count, then scatter).
//
// CTA b takes the medium segments b, b + G, b + 2G, ... (G CTAs), so it knows
// its next segment in advance: the next segment's offsets are loaded during
// the current count pass, and its tiles are requested while the current
// segment is scattered -- a tile slot as soon as the current segment's tile
// in it has been taken into registers, the slots the current segment does not
// use at once.  The loads of one segment thus overlap the scatter of the one
// before.  A slab of two tiles keeps the kernel at four CTAs per SM (a slab of
// four at two CTAs per SM was slower: the tile step needs the occupancy).
//
// Measured (100,000 LogNormal(ln 1024, 1.5) segments, u32, m = 4): the
// segments of two tiles take 165 us here against 152 us less in the run
// kernels, so the single read does not pay for itself there -- the tile step,
// not the re-read, bounds those segments (a segment of ~1.5 tiles costs two
// tile steps either way).  It stays a tuned option (mid_tiles) and is off by
// default.
template <class V, int M, int THREADS, int KMAX>
struct MidSmem {
    using G = TileGeom<V, THREADS, M>;
    static constexpr size_t kSlabBytes = static_cast<size_t>(KMAX) * G::kTile * sizeof(V);
    static constexpr size_t kBytes = 1024 + kSlabBytes + G::kStageBytes + G::kCntBytes;
};

template <class V, class D, int M, int THREADS, int KMAX>
__global__ void __launch_bounds__(THREADS, 4)
    seg_mid(SegArgs a, D d, const __grid_constant__ CUtensorMap tmap) {
    using L = MidSmem<V, M, THREADS, KMAX>;
    using TG = typename L::G;
    constexpr int ITEMS = TG::kItems;
    constexpr int P = TG::kTile;
    constexpr int ROWS = TG::kRows;
    constexpr uint32_t AU = TG::kAU;
    constexpr int W = THREADS / 32;
    constexpr uint32_t kPerRow = 128u / sizeof(V);
    static_assert(M <= 16 && M >= 2, "class bound");
    static_assert(KMAX >= 2 && KMAX <= 32, "one phase bit per slab tile");
    static_assert(ROWS <= 256, "TMA box height");

    extern __shared__ __align__(128) unsigned char smem_raw[];
    const uint32_t raw = smem_addr(smem_raw);
    unsigned char* base = smem_raw + (((raw + 1023u) & ~1023u) - raw);
    V* slab = reinterpret_cast<V*>(base);
    V* stage = reinterpret_cast<V*>(base + L::kSlabBytes);
    uint32_t* cnt_sm = reinterpret_cast<uint32_t*>(base + L::kSlabBytes + TG::kStageBytes);

    __shared__ __align__(8) uint64_t bars[KMAX];
    __shared__ TileShared<M> sh;
    __shared__ uint32_t red[W][M];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const V* in = static_cast<const V*>(a.in);
    V* out = static_cast<V*>(a.out);
    const uint32_t out_phase =
        static_cast<uint32_t>(reinterpret_cast<uintptr_t>(out) / sizeof(V)) & (AU - 1u);
    const bool tma_ok = a.use_tma != 0;
    const uint64_t map_elems = (a.n * sizeof(V) / 128u) * kPerRow;
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t num_mids = a.hdr->num_mids;
    const uint32_t G = gridDim.x;
    const uint32_t e0 = tid * ITEMS;
    uint32_t parity = 0;  // bit i: the phase of bars[i] that completes next

    // A segment's element range and its tiles from the 128-byte row of a0 (at
    // most mid_tiles <= KMAX by the planner's classification).
    struct Seg {
        uint64_t a0, a1, rb;
        uint32_t s, ntiles;
    };
    auto make_seg = [&](uint32_t s, uint64_t a0, uint64_t a1) {
        Seg g;
        g.s = s;
        g.a0 = a0;
        g.a1 = a1;
        g.rb = a0 & ~static_cast<uint64_t>(kPerRow - 1u);
        g.ntiles = static_cast<uint32_t>(
            min((a1 - g.rb + P - 1u) / P, static_cast<uint64_t>(KMAX)));
        return g;
    };
    // a tile comes by TMA when the segment's part of it lies inside the
    // tensor map (the input's whole 128-byte rows; rows past the map read as
    // zeros and lie outside the segment)
    auto via_tma = [&](const Seg& g, uint32_t i) {
        return tma_ok && min(g.a1, g.rb + static_cast<uint64_t>(i + 1) * P) <= map_elems;
    };
    auto issue = [&](const Seg& g, uint32_t i) {  // tile i of g into slab slot i
        if (via_tma(g, i)) {
            mbar_arrive_expect_tx(&bars[i], P * sizeof(V));
            tma_load_2d(slab + static_cast<size_t>(i) * P, &tmap, 0,
                        static_cast<int32_t>(g.rb / kPerRow + static_cast<uint64_t>(i) * ROWS),
                        &bars[i]);
        } else {
            mbar_arrive(&bars[i]);
        }
    };
    auto range = [&](const Seg& g, uint32_t i, uint32_t& lo, uint32_t& hi) {
        const uint64_t ts = g.rb + static_cast<uint64_t>(i) * P;
        lo = static_cast<uint32_t>(max(g.a0, ts) - ts);
        hi = static_cast<uint32_t>(min(g.a1, ts + P) - ts);
    };
    auto take = [&](const Seg& g, uint32_t i, uint32_t lo, uint32_t hi, V (&v)[ITEMS]) {
        if (via_tma(g, i)) {
            take_swizzled<V, ITEMS>(slab + static_cast<size_t>(i) * P, v);
        } else {
            const uint64_t ts = g.rb + static_cast<uint64_t>(i) * P;
#pragma unroll
            for (int q = 0; q < ITEMS; q++)
                v[q] = (e0 + q >= lo && e0 + q < hi) ? in[ts + e0 + q] : V();
        }
    };

    if (tid == 0) {
#pragma unroll
        for (int q = 0; q < KMAX; q++) mbar_init(&bars[q], 1);
        mbar_fence_init();
    }
    __syncthreads();

    uint32_t t = blockIdx.x;
    if (t >= num_mids) return;
    Seg cur;
    {
        const uint32_t s = a.mids[t];
        cur = make_seg(s, a.offsets[s], a.offsets[s + 1]);
    }
    if (tid == 0)
        for (uint32_t i = 0; i < cur.ntiles; i++) issue(cur, i);
    // the segment after the next one: its index is loaded one iteration early
    uint32_t s_next = t + G < num_mids ? a.mids[t + G] : 0u;

    for (; t < num_mids; t += G) {
        const bool has_next = t + G < num_mids;
        uint64_t n0 = 0, n1 = 0;
        if (has_next) {  // used after the count pass
            n0 = a.offsets[s_next];
            n1 = a.offsets[s_next + 1];
        }
        const uint32_t s_after = t + 2u * G < num_mids ? a.mids[t + 2u * G] : 0u;
        const D dj = seg_discr(a, d, seg_classes(a, cur.s));

        // ---- count pass: lane c of every warp keeps the warp's count of class c
        uint32_t wt = 0;
        bool ok = true;
        for (uint32_t i = 0; i < cur.ntiles; i++) {
            ok = mbar_wait_bounded(&bars[i], (parity >> i) & 1u) && ok;
            uint32_t lo, hi;
            range(cur, i, lo, hi);
            const bool full = lo == 0u && hi == static_cast<uint32_t>(P);
            V v[ITEMS];
            take(cur, i, lo, hi, v);
            NibbleCounts<M> nc;
            nc.init();
            uint32_t last_c = M;  // element 15 stays out of the nibbles (a nibble holds 15)
#pragma unroll
            for (int j = 0; j < ITEMS; j++) {
                if (full || (e0 + j >= lo && e0 + j < hi)) {
                    const uint32_t c = dj(v[j]);
                    if (j < 15) nc.inc(c); else last_c = c;
                }
            }
#pragma unroll
            for (int c = 0; c < M; c++) {
                const uint32_t x = __reduce_add_sync(
                    0xffffffffu, nc.get(c) + (last_c == static_cast<uint32_t>(c) ? 1u : 0u));
                if (lane == c) wt += x;
            }
        }
        if (lane < M) red[warp][lane] = wt;
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicOr(&a.hdr->error, kErrTimeout);
                for (uint32_t i = 0; i < cur.ntiles; i++)  // copies still in flight
                    (void)mbar_wait_bounded(&bars[i], (parity >> i) & 1u);
            }
            break;
        }
        parity ^= cur.ntiles >= 32u ? 0xffffffffu : ((1u << cur.ntiles) - 1u);
        Seg nxt{};
        if (has_next) nxt = make_seg(s_next, n0, n1);

        // ---- the segment's class totals: sizes, head flags, cursors
        if (warp == 0) {
            uint32_t tot = 0;
            if (lane < M) {
#pragma unroll
                for (int w = 0; w < W; w++) tot += red[w][lane];
            }
            const uint32_t excl = warp_incl_scan(tot) - tot;
            if (lane < M) {
                sh.cursor[0][lane] = static_cast<uint32_t>(cur.a0) + excl;
                if (a.seg_sizes != nullptr && static_cast<uint32_t>(lane) < a.m)
                    a.seg_sizes[static_cast<uint64_t>(cur.s) * a.m + lane] = tot;
                if (a.headflags != nullptr && tot > 0) a.headflags[cur.a0 + excl] = tot;
            }
            // the next segment's tiles in the slots this one leaves unused
            if (lane == 0 && has_next)
                for (uint32_t i = cur.ntiles; i < nxt.ntiles; i++) issue(nxt, i);
        }
        __syncthreads();

        // ---- scatter pass from the slab; slot i takes the next segment's tile
        // i once this segment's tile i is in registers
        for (uint32_t i = 0; i < cur.ntiles; i++) {
            uint32_t lo, hi;
            range(cur, i, lo, hi);
            const bool full = lo == 0u && hi == static_cast<uint32_t>(P);
            V v[ITEMS];
            take(cur, i, lo, hi, v);
            auto refill = [&] {
                if (tid == 0 && has_next && i < nxt.ntiles) issue(nxt, i);
            };
            if constexpr (M == 2)
                (void)tile_filter<V, D, THREADS, true>(dj, v, lo, hi, full, stage, cnt_sm, sh, i & 1u,
                                                       OutFlat<V>{out, out_phase}, true, refill);
            else
                (void)tile_scatter<V, D, M, THREADS, true, false>(dj, v, lo, hi, full, stage, cnt_sm, sh,
                                                           i & 1u, OutFlat<V>{out, out_phase}, true,
                                                           refill);
        }
        cur = nxt;
        s_next = s_after;
    }
    if (tid < M) bulk_wait_all();
}

// ------------------------------------------------ head flags -> offsets --
// The reference's segment descriptor (MdiscrSegmHost.cu.h:36-42,
// populateSizesArray HelpersCommon.h:105-151) is an n-entry array holding each
// segment's length at its first element and 0 elsewhere.  Two launches turn it
// into offsets[0..S] and S (in the header); the planner then checks that every
// flag equals the distance to the next start.
//
//   seg_flags_stage    a warp per chunk reads its flags once, eight 16-byte words a
//                      lane in flight, and writes the positions of its non-zero
//                      flags in order into the chunk's part of a staging array
//                      (stage[chunk start + j]) and their number; the last CTA to
//                      finish (ticket, no waiting) scans the chunk counts into
//                      chunk prefixes, S and offsets[S] = n.
//   seg_flags_compact  a warp per chunk moves its staged positions to
//                      offsets[prefix + j].
//
// Flags are sparse (a segment has one): a word of all lanes without one costs a
// vote.  No CTA waits on another, and no warp on its CTA before the end.  10^8 flags,
// stage and compaction: 90 us when CTAs read tiles of 4096 flags with two barriers
// each, 84 now (the read alone at the copy rate: 61).
constexpr uint32_t kMaxFlagChunks = 4096;

struct FlagsArgs {
    const int32_t* flags;
    uint64_t n;
    uint64_t chunk;      // flags per chunk (a multiple of 128)
    uint32_t* stage;     // [n] staged start positions, chunk k's from k * chunk
    uint32_t* cnt;       // [chunks] start positions per chunk
    uint32_t* pre;       // [chunks] exclusive prefix of cnt
    uint64_t* offsets;   // [S + 1]
    SegHeader* hdr;
};

template <int THREADS>
__global__ void __launch_bounds__(THREADS) seg_flags_stage(FlagsArgs fa) {
    constexpr int W = THREADS / 32;
    constexpr int U = 8;
    constexpr int PER = static_cast<int>(kMaxFlagChunks) / THREADS;
    __shared__ uint32_t warp_tot[W];
    __shared__ int last_sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_launch_dependents();
    const uint32_t k = blockIdx.x * W + warp;
    const uint64_t c0 = min(static_cast<uint64_t>(k) * fa.chunk, fa.n);
    const uint64_t c1 = min(c0 + fa.chunk, fa.n);
    uint32_t* out = fa.stage + c0;
    bool bad = false;
    // four flags a lane, in order over the lanes: positions of the non-zero ones
    auto take = [&](const int4& f, uint64_t e) {
        const uint32_t nz = (f.x != 0 ? 1u : 0u) | (f.y != 0 ? 2u : 0u) | (f.z != 0 ? 4u : 0u) |
                            (f.w != 0 ? 8u : 0u);
        if (__ballot_sync(0xffffffffu, nz != 0u) == 0u) return;
        bad |= (f.x | f.y | f.z | f.w) < 0;
        const uint32_t c = static_cast<uint32_t>(__popc(nz));
        const uint32_t incl = warp_incl_scan(c);
        uint32_t* p = out + (incl - c);
#pragma unroll
        for (uint32_t q = 0; q < 4; q++)
            if (nz >> q & 1u) *p++ = static_cast<uint32_t>(e + q);
        out += __shfl_sync(0xffffffffu, incl, 31);
    };
    uint64_t e = c0 + 4u * lane;
    if ((reinterpret_cast<uintptr_t>(fa.flags) & 15u) == 0) {
        for (; e - 4u * lane + 128u * U <= c1; e += 128u * U) {
            int4 f[U];
#pragma unroll
            for (int u = 0; u < U; u++) f[u] = __ldg(reinterpret_cast<const int4*>(fa.flags + e + 128u * u));
            int any = 0;
#pragma unroll
            for (int u = 0; u < U; u++) any |= f[u].x | f[u].y | f[u].z | f[u].w;
            if (__ballot_sync(0xffffffffu, any != 0) == 0u) continue;
#pragma unroll
            for (int u = 0; u < U; u++) take(f[u], e + 128u * u);
        }
    }
    for (; e - 4u * lane < c1; e += 128u) {  // the rest, and all of unaligned flags
        int4 f;
        f.x = e < c1 ? __ldg(fa.flags + e) : 0;
        f.y = e + 1u < c1 ? __ldg(fa.flags + e + 1u) : 0;
        f.z = e + 2u < c1 ? __ldg(fa.flags + e + 2u) : 0;
        f.w = e + 3u < c1 ? __ldg(fa.flags + e + 3u) : 0;
        take(f, e);
    }
    if (bad) atomicOr(&fa.hdr->error, kErrSegments);
    if (lane == 0) fa.cnt[k] = static_cast<uint32_t>(out - (fa.stage + c0));
    __threadfence();
    __syncthreads();
    if (tid == 0) last_sh = (atomicAdd(&fa.hdr->flags_done, 1u) == gridDim.x - 1u);
    __syncthreads();
    if (!last_sh) return;
    __threadfence();
    // last CTA: exclusive scan of the chunk counts, S, offsets[S]
    const uint32_t chunks = gridDim.x * W;
    uint32_t x[PER], sum = 0;
#pragma unroll
    for (int q = 0; q < PER; q++) {
        const uint32_t b = static_cast<uint32_t>(tid) * PER + q;
        x[q] = b < chunks ? __ldcg(&fa.cnt[b]) : 0u;
        sum += x[q];
    }
    const uint32_t incl = warp_incl_scan(sum);
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    uint32_t before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < W; w++) {
        before += w < warp ? warp_tot[w] : 0u;
        all += warp_tot[w];
    }
    uint32_t run = before + incl - sum;
#pragma unroll
    for (int q = 0; q < PER; q++) {
        const uint32_t b = static_cast<uint32_t>(tid) * PER + q;
        if (b < chunks) fa.pre[b] = run;
        run += x[q];
    }
    if (tid == 0) {
        fa.hdr->num_segs = all;
        fa.offsets[all] = fa.n;
        if (fa.n > 0 && __ldg(fa.flags) == 0) atomicOr(&fa.hdr->error, kErrSegments);
        fa.hdr->flags_done = 0u;  // for the next call
    }
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS) seg_flags_compact(FlagsArgs fa) {
    pdl_wait();
    const uint32_t w = blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5);
    const uint64_t c0 = min(static_cast<uint64_t>(w) * fa.chunk, fa.n);
    const uint32_t k = fa.cnt[w], p = fa.pre[w];
    for (uint32_t j = threadIdx.x & 31u; j < k; j += 32u) fa.offsets[p + j] = fa.stage[c0 + j];
}

}  // namespace mdx
