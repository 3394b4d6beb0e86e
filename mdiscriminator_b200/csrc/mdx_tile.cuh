// mdx_tile.cuh -- the per-tile rank / stage / write-out step shared by the
// plain scatter kernel and the segmented scatter items (m <= 16).
//
// A tile is THREADS * ITEMS elements (BPT = 64 or 32 contiguous bytes per
// thread: two tile geometries, chosen per call by the tuning table).  For
// the elements of tile-local range [lo, hi):
//  * pass 1: each thread counts its own consecutive elements per class with
//    4-bit counters in a register (the 16th element is kept aside so no lane can
//    reach 16) and publishes the counts to a matrix of 16-bit pairs;
//  * row scans: warp w < m/2 scans word row w of the matrix, two classes at once
//    (exclusive prefix over threads = stable order); those warps derive the
//    tile's class runs (lanes = classes) and fold each run's stage slot into
//    their rows;
//  * pass 2: element -> stage slot = row prefix + local rank; m < 16 keeps the
//    ranks of pass 1 in registers, m = 16 lets the thread's entry of the matrix
//    move on with every element (a 64-bit shift less per element, against a
//    store: N = 2^28 u32, 512 threads: scatter 391 against 444 us, but 383
//    against 353 at m = 8, where the shifts are cheap and the chain is not);
//  * write-out: each class run sits in the stage at the same 16-byte phase as
//    its destination, so its aligned interior leaves by one bulk store
//    (cp.async.bulk shared -> global) and threads store the < 16-byte head and
//    tail.  Before the stage is rewritten the previous bulk stores must have
//    read it (cp.async.bulk.wait_group.read).
#pragma once

#include <type_traits>

#include "mdx_device.cuh"

namespace mdx {

// Per-thread class counters in 4-bit lanes: one u32 holds 8 classes, two
// hold 16.
template <int M>
struct NibbleCounts {
    static_assert(M <= 16, "nibble counters cover at most 16 classes");
    static constexpr int NW = (M + 7) / 8;
    uint32_t w[NW];
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int q = 0; q < NW; q++) w[q] = 0;
    }
    __device__ __forceinline__ uint32_t get(uint32_t c) const {
        if constexpr (NW == 1) {
            return (w[0] >> (c << 2)) & 15u;
        } else {  // sixteen nibbles: one 64-bit shift
            const uint64_t x = (static_cast<uint64_t>(w[1]) << 32) | w[0];
            return static_cast<uint32_t>(x >> (c << 2)) & 15u;
        }
    }
    __device__ __forceinline__ void inc(uint32_t c) {
        if constexpr (NW == 1) {
            w[0] += 1u << (c << 2);
        } else {
            uint64_t x = (static_cast<uint64_t>(w[1]) << 32) | w[0];
            x += 1ull << (c << 2);
            w[0] = static_cast<uint32_t>(x);
            w[1] = static_cast<uint32_t>(x >> 32);
        }
    }
};

template <class V>
__device__ __forceinline__ void unpack16_to(const uint4& r, V* e);
template <>
__device__ __forceinline__ void unpack16_to<uint32_t>(const uint4& r, uint32_t* e) {
    e[0] = r.x; e[1] = r.y; e[2] = r.z; e[3] = r.w;
}
template <>
__device__ __forceinline__ void unpack16_to<uint64_t>(const uint4& r, uint64_t* e) {
    e[0] = static_cast<uint64_t>(r.x) | (static_cast<uint64_t>(r.y) << 32);
    e[1] = static_cast<uint64_t>(r.z) | (static_cast<uint64_t>(r.w) << 32);
}
template <>
__device__ __forceinline__ void unpack16_to<Rec16>(const uint4& r, Rec16* e) {
    e[0].w[0] = r.x; e[0].w[1] = r.y; e[0].w[2] = r.z; e[0].w[3] = r.w;
}

template <class V, int THREADS, int M, int BPT = 64>
struct TileGeom {
    static_assert(BPT == 64 || BPT == 32 || BPT == 16, "64, 32 or 16 bytes per thread");
    static constexpr int kItems = BPT / static_cast<int>(sizeof(V));  // BPT bytes per thread
    static constexpr int kTile = THREADS * kItems;
    static constexpr int kRows = kTile * static_cast<int>(sizeof(V)) / 128;  // 128-byte rows
    static constexpr uint32_t kAU = 16 / sizeof(V);                 // elements per 16 bytes
    // every class run gets kAU slots of slack for its 16-byte phase
    static constexpr int kStageElems = kTile + static_cast<int>(kAU) * M;
    static constexpr size_t kStageBytes = static_cast<size_t>(kStageElems) * sizeof(V);
    // m <= 16: [class pair][thread] words of two 16-bit counts; more classes:
    // [class / 4][thread] words of four byte counts and a table of up to 32 rows
    // (tile_scatter_bytes)
    static constexpr size_t kCntBytes = M > 16
                                            ? static_cast<size_t>(M) * THREADS + 32 * (M + 4) * 2
                                            : static_cast<size_t>(M) * THREADS * 2;
    static_assert(kStageElems < 65536, "stage slots are kept in 16 bits");
};

// Shared-memory state of the tile step.
template <int M>
struct TileShared {
    uint32_t cursor[2][M];  // ping-pong by tile parity
    uint32_t run_start[M], run_cnt[M], run_dst[M];
    alignas(16) uint32_t rowtot[M];
};

// Where a tile's class runs go.  `idx` is an element's position in the whole
// output (< 2^32).
//
// OutFlat: one array.  phase = (out / sizeof(V)) mod (16 / sizeof(V)).
template <class V>
struct OutFlat {
    static constexpr uint32_t kAU = 16 / sizeof(V);  // elements a bulk store is aligned to
    V* out;
    uint32_t phase_;
    __device__ __forceinline__ uint32_t phase() const { return phase_; }
    __device__ __forceinline__ V* at(uint32_t idx) const { return out + idx; }
    // End of the piece [idx, end) that lies in one buffer.
    __device__ __forceinline__ uint32_t piece_end(uint32_t, uint32_t end) const { return end; }
};

// OutSharded: the output is cut into R chunks that live in different buffers
// (one per rank, typically on other GPUs, reached through peer mappings):
// chunk q holds positions [q * chunk, (q + 1) * chunk) (trailing chunks may
// be short or empty), the last chunk everything from (R - 1) * chunk on.
// Every chunk pointer is 16-byte aligned and `chunk` is a multiple of
// 16 / sizeof(V) elements, so a position's 16-byte phase is the same in every
// chunk and a run that crosses a chunk boundary splits into pieces that each
// stay bulk-store aligned.
constexpr int kMaxRanks = 128;
template <class V>
struct OutSharded {
    static constexpr uint32_t kAU = 16 / sizeof(V);
    V* chunks[kMaxRanks];
    uint32_t chunk;
    uint32_t R;
    __device__ __forceinline__ uint32_t phase() const { return 0u; }
    __device__ __forceinline__ V* at(uint32_t idx) const {
        const uint32_t q = min(idx / chunk, R - 1u);
        return chunks[q] + (idx - q * chunk);
    }
    __device__ __forceinline__ uint32_t piece_end(uint32_t idx, uint32_t end) const {
        const uint32_t q = idx / chunk;
        if (q + 1u >= R) return end;
        const uint64_t b = static_cast<uint64_t>(q + 1u) * chunk;
        return b < end ? static_cast<uint32_t>(b) : end;
    }
};

// OutRows: the tile's order is wanted, not its elements: runs lie in the stage one
// after another without room for a 16-byte phase, and run_dst holds what has to be
// added to a slot to give its position in the output (mdx_rows.cuh).
struct OutRows {
    static constexpr uint32_t kAU = 1;
    __device__ __forceinline__ uint32_t phase() const { return 0u; }
};

// Take a thread's ITEMS * sizeof(V) (64 or 32) bytes of a tile that TMA
// placed in shared memory with the 128-byte swizzle (16-byte chunk q of
// 128-byte row r sits at chunk q ^ (r & 7)).
template <class V, int ITEMS>
__device__ __forceinline__ void take_swizzled(const V* tile, V (&v)[ITEMS]) {
    constexpr uint32_t AU = 16 / sizeof(V);
    constexpr uint32_t BPT = ITEMS * sizeof(V);
    static_assert(BPT == 64 || BPT == 32, "64 or 32 bytes per thread");
    constexpr uint32_t TPR = 128 / BPT, CPT = BPT / 16;  // threads per row, chunks per thread
    const unsigned char* tb = reinterpret_cast<const unsigned char*>(tile);
    const uint32_t row = threadIdx.x / TPR;
#pragma unroll
    for (uint32_t q = 0; q < CPT; q++) {
        const uint32_t chunk = ((threadIdx.x % TPR) * CPT + q) ^ (row & 7u);
        const uint4 r = *reinterpret_cast<const uint4*>(tb + row * 128u + chunk * 16u);
        unpack16_to<V>(r, &v[q * AU]);
    }
}

// A warp whose elements all belong to one class (sorted or clustered input)
// fills 32 * ITEMS consecutive stage slots from `run` on, ITEMS from each lane.
// Stored lane by lane, the lanes would be ITEMS slots apart and hit two banks in
// all; so each lane stores its slots in an order of its own (slot j ^ lane / 2),
// which spreads a store over the banks, and the warp then puts the slots of
// every 32 in order.  Three conflict-free accesses an element instead of one that
// is repeated for each of 16 lanes (4-byte elements) of a bank: N = 2^28 u32
// sorted by class, scatter at m = 2, 8, 16: 601, 652, 733 us before, 333, 349,
// 365 with it.
template <class V, int ITEMS>
__device__ __forceinline__ void place_warp_run(V* run, const V (&v)[ITEMS]) {
    const uint32_t lane = threadIdx.x & 31u;
    constexpr uint32_t I = ITEMS;
#pragma unroll
    for (uint32_t j = 0; j < I; j++) run[I * lane + (j ^ ((lane >> 1) & (I - 1u)))] = v[j];
    __syncwarp();
#pragma unroll 4
    for (uint32_t k = 0; k < I; k++) {  // slots 32 k ..: in order; they stay among themselves
        const uint32_t l = 32u / I * k + lane / I;  // the lane slot 32 k + lane came from
        const V x = run[I * l + ((lane % I) ^ ((l >> 1) & (I - 1u)))];
        __syncwarp();
        run[32u * k + lane] = x;
    }
}

// The same where lanes of one class each (`one`) lie beside others: each such lane has
// stored its ITEMS consecutive slots from `run` on in its own order (slot
// j ^ spread_of(lane)), and the warp puts them in order.
template <int ITEMS>
__device__ __forceinline__ uint32_t spread_of(uint32_t lane) {
    return (lane >> 1) & (ITEMS - 1u);
}
template <class V, int ITEMS>
__device__ __forceinline__ void order_lane_runs(V* stage, bool one, uint32_t run) {
    const uint32_t lane = threadIdx.x & 31u;
    constexpr uint32_t I = ITEMS, kNone = 0xffffffffu;
    __syncwarp();
#pragma unroll
    for (uint32_t k = 0; k < I; k++) {  // 32 / I lanes' slots at a time; they stay among themselves
        const uint32_t l = 32u / I * k + lane / I;
        const uint32_t r = __shfl_sync(0xffffffffu, one ? run : kNone, l);
        V x;
        if (r != kNone) x = stage[r + ((lane % I) ^ spread_of<ITEMS>(l))];
        __syncwarp();
        if (r != kNone) stage[r + lane % I] = x;
    }
}

// Whether the warp's lanes all have `one` (their elements share a class) and the
// same class c.
__device__ __forceinline__ bool warp_of_one_class(bool one, uint32_t c) {
    const uint32_t c0 = __shfl_sync(0xffffffffu, c, 0);  // by every lane, whatever `one` says
    return __all_sync(0xffffffffu, one && c == c0);
}

// Count matrix of the nibble step: a 32-bit word holds the 16-bit counts of two
// classes and a row one word of every thread, so a warp's words of a row lie in
// 32 banks whatever classes its lanes look up (16-bit entries side by side put
// two threads in a bank and cost two wavefronts a lookup).  Thread t = PER g +
// 4 h + i (PER = threads a scan lane takes) has column 128 h + ((4 g + i) ^ X h):
// a scan lane's PER words are then 16-byte loads that are consecutive over the
// lanes.
template <int THREADS>
struct CountColumns {
    static constexpr uint32_t kPer = THREADS / 32;
    static constexpr uint32_t kX = 128u / kPer;  // 32 banks over the kPer / 4 loads
    static_assert(kPer == 8 || kPer == 16, "row scans load 8 or 16 words per lane");
    static __device__ __forceinline__ uint32_t column(uint32_t t) {
        const uint32_t g = t / kPer, h = (t / 4u) % (kPer / 4u), i = t % 4u;
        return 128u * h + ((4u * g + i) ^ (kX * h));
    }
    // first word of scan lane l's load h
    static __device__ __forceinline__ uint32_t chunk(uint32_t l, uint32_t h) {
        return 128u * h + ((4u * l) ^ (kX * h));
    }
};

// Discriminators that are as cheap to evaluate twice as to remember.
template <class D>
struct CheapClass : std::is_same<D, DiscrMask> {};

// Per-thread class counts of the nibble step and where class c's 16-bit count
// lies: classes k and k + M / 2 share word k.
template <int M>
struct ThreadCounts {
    static_assert(M == 4 || M == 8 || M == 16, "class bound");
    static constexpr int kRows = M / 2;
    static constexpr uint32_t kHalf = M / 2;
    // four classes: 8-bit counters, which hold the 16th element too
    static constexpr bool kNibbles = M > 4;
    uint32_t w[2];
    __device__ __forceinline__ void init() { w[0] = w[1] = 0; }
    __device__ __forceinline__ uint32_t get(uint32_t c) const {
        if constexpr (M == 4) return (w[0] >> (c << 3)) & 0xffu;
        else if constexpr (M == 8) return (w[0] >> (c << 2)) & 15u;
        else return static_cast<uint32_t>(((static_cast<uint64_t>(w[1]) << 32) | w[0]) >> (c << 2)) & 15u;
    }
    __device__ __forceinline__ void inc(uint32_t c) {
        if constexpr (M == 4) {
            w[0] += 1u << (c << 3);
        } else if constexpr (M == 8) {
            w[0] += 1u << (c << 2);
        } else {  // sixteen nibbles: one 64-bit shift
            uint64_t x = (static_cast<uint64_t>(w[1]) << 32) | w[0];
            x += 1ull << (c << 2);
            w[0] = static_cast<uint32_t>(x);
            w[1] = static_cast<uint32_t>(x >> 32);
        }
    }
    // the counts of classes r (low half) and r + M / 2
    __device__ __forceinline__ uint32_t word(int r) const {
        if constexpr (M == 4) return (w[0] >> (8 * r)) & 0x00ff00ffu;
        else if constexpr (M == 8) return (w[0] >> (4 * r)) & 0x000f000fu;
        else return (__byte_perm(w[0], w[1], r < 4 ? 0x5410 : 0x7632) >> (4 * (r & 3))) & 0x000f000fu;
    }
    // byte offset of class c's count from the thread's column
    template <int THREADS>
    static __device__ __forceinline__ uint32_t offset(uint32_t c) {
        constexpr uint32_t kRow = 4u * THREADS;
        return c * kRow - c / kHalf * (kHalf * kRow - 2u);
    }
};

// What run_dst of a run says: its position in the output, or (OutRows) the
// distance from its stage slots to it.
template <class OUT>
__device__ __forceinline__ uint32_t run_position(uint32_t dst, uint32_t st) {
    return std::is_same<OUT, OutRows>::value ? dst - st : dst;
}

// Write-out of a tile whose class runs lie in the stage, each at its destination's
// 16-byte phase: a bulk store of each run's aligned interior; threads store the
// unaligned heads and tails (those of warp 0, which issue the bulk stores, only
// when the others do not suffice).
template <class V, int M, int THREADS, class OUT>
__device__ __forceinline__ void write_runs(const V* stage, const TileShared<M>& sh, const OUT& out) {
    constexpr uint32_t AU = OUT::kAU;
    constexpr int kEdges = M * 2 * static_cast<int>(AU);  // head and tail elements at most
    constexpr int kFirst = M <= 32 && 32 + kEdges <= THREADS ? 32 : 0;
    const int tid = threadIdx.x;
    if (tid < M) {
        const uint32_t s = sh.run_start[tid], cc = sh.run_cnt[tid];
        uint32_t head = (AU - (s & (AU - 1u))) & (AU - 1u);
        if (head > cc) head = cc;
        const uint32_t body = ((cc - head) / AU) * AU;
        uint32_t a0 = sh.run_dst[tid] + head, sl = s + head;
        const uint32_t a1 = a0 + body;
        while (a0 < a1) {  // one piece per destination buffer
            const uint32_t b = out.piece_end(a0, a1);
            bulk_store_s2g(out.at(a0), stage + sl, (b - a0) * sizeof(V));
            sl += b - a0;
            a0 = b;
        }
        bulk_commit();
    }
    if constexpr (AU > 1) {
#pragma unroll
        for (int t0 = 0; t0 < kEdges; t0 += THREADS) {
            const int t = tid - kFirst + t0;
            if (t < 0 || t >= kEdges) continue;
            const uint32_t c = static_cast<uint32_t>(t) / (2 * AU), q = static_cast<uint32_t>(t) % (2 * AU);
            const uint32_t s = sh.run_start[c], cc = sh.run_cnt[c];
            uint32_t head = (AU - (s & (AU - 1u))) & (AU - 1u);
            if (head > cc) head = cc;
            const uint32_t body = ((cc - head) / AU) * AU;
            uint32_t off = 0xffffffffu;
            if (q < AU) {
                if (q < head) off = q;
            } else if (head + body + (q - AU) < cc) {
                off = head + body + (q - AU);
            }
            if (off != 0xffffffffu) *out.at(sh.run_dst[c] + off) = stage[s + off];
        }
    }
}

// One tile: see the file comment.  `full` means lo == 0 and hi == TILE (no
// bounds checks).  FORWARD: run c of this tile starts at cursor[par][c] and
// the cursor advances; otherwise it ends there and the cursor moves back.
// `after_counts` runs right after the first barrier (the input ring slot is
// consumed by then).  Returns false, having written nothing, when `ok` is
// false on any thread.
template <class V, class D, int M, int THREADS, bool FORWARD, bool CLUSTERED, class OUT,
          class AfterCounts, int ITEMS>
__device__ __forceinline__ bool tile_scatter(const D& d, const V (&v)[ITEMS], uint32_t lo,
                                             uint32_t hi, bool full, V* stage, uint32_t* cnt_sm,
                                             TileShared<M>& sh, uint32_t par, const OUT& out,
                                             bool ok, AfterCounts after_counts) {
    using G = TileGeom<V, THREADS, M, ITEMS * static_cast<int>(sizeof(V))>;
    static_assert(G::kItems == ITEMS, "geometry");
    using CC = CountColumns<THREADS>;
    using TC = ThreadCounts<M>;
    constexpr uint32_t AU = OUT::kAU;
    constexpr int W = THREADS / 32;
    constexpr int PER = static_cast<int>(CC::kPer);
    static_assert(TC::kRows <= W, "a warp per row");
    static_assert(ITEMS == 16 || ITEMS == 8 || ITEMS == 4 || ITEMS == 2, "thread elements");
    // a nibble holds 15: the 16th element is kept out of them
    constexpr int kIn = TC::kNibbles && ITEMS > 15 ? 15 : ITEMS;
    constexpr bool kRanks = M < 16;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t e0 = tid * ITEMS;
    unsigned char* my_cnt = reinterpret_cast<unsigned char*>(cnt_sm + CC::column(tid));
    auto count_at = [&](uint32_t c) -> uint16_t& {
        return *reinterpret_cast<uint16_t*>(my_cnt + TC::template offset<THREADS>(c));
    };

    // ---- pass 1
    TC tc;
    tc.init();
    uint32_t last_c = M;  // class of the element kept out of the nibbles
    uint32_t lr[kRanks ? (ITEMS + 7) / 8 : 1];  // local ranks, four bits each
    if constexpr (kRanks) {
#pragma unroll
        for (int q = 0; q < (ITEMS + 7) / 8; q++) lr[q] = 0;
    }
    // classes kept for pass 2 where working them out again costs more (a byte each;
    // m <= 8 has no registers to spare for them)
    constexpr bool kKeep = M == 16 && !CheapClass<D>::value;
    uint32_t kept[kKeep ? (ITEMS + 3) / 4 : 1];
    if constexpr (kKeep) {
#pragma unroll
        for (int q = 0; q < (ITEMS + 3) / 4; q++) kept[q] = 0;
    }
    auto class_of = [&](int j) -> uint32_t {
        if constexpr (kKeep) return __byte_perm(kept[j >> 2], 0u, 0x4440 + (j & 3));
        else return d(v[j]);
    };
    auto count = [&](int j) {
        const uint32_t c = d(v[j]);
        if constexpr (kKeep) kept[j >> 2] += c << (8 * (j & 3));
        if constexpr (kRanks) lr[j >> 3] += tc.get(c) << (4 * (j & 7));
        if (j < kIn) tc.inc(c); else last_c = c;
    };
    if (full) {
#pragma unroll
        for (int j = 0; j < ITEMS; j++) count(j);
    } else {
#pragma unroll
        for (int j = 0; j < ITEMS; j++)
            if (e0 + j >= lo && e0 + j < hi) count(j);
    }
    const uint32_t c_last = class_of(ITEMS - 1);
    bool one_class = false;  // the warp's elements
    if constexpr (CLUSTERED) one_class = full && warp_of_one_class(tc.get(c_last) == kIn, c_last);
#pragma unroll
    for (int r = 0; r < TC::kRows; r++)
        *reinterpret_cast<uint32_t*>(my_cnt + r * 4 * THREADS) = tc.word(r);
    if constexpr (kIn < ITEMS)
        if (last_c < static_cast<uint32_t>(M)) count_at(last_c) += 1;
    if (__syncthreads_or(!ok)) return false;  // (A)
    after_counts();

    // ---- row scans: warp w < M/2 scans row w, two classes at once (a class's
    // sum is at most the tile, < 2^16); the other warps idle here
    const bool scans = warp < TC::kRows;
    uint32_t* row = cnt_sm + warp * THREADS;
    uint32_t pre[PER];  // packed exclusive prefixes of this lane's threads
    if (scans) {
        uint32_t x[PER];
#pragma unroll
        for (int u = 0; u < PER / 4; u++) {
            const uint4 a = *reinterpret_cast<const uint4*>(row + CC::chunk(lane, u));
            x[4 * u + 0] = a.x;
            x[4 * u + 1] = a.y;
            x[4 * u + 2] = a.z;
            x[4 * u + 3] = a.w;
        }
        uint32_t tot = 0;
#pragma unroll
        for (int q = 0; q < PER; q++) tot += x[q];
        const uint32_t incl = warp_incl_scan(tot);
        uint32_t run = incl - tot;
#pragma unroll
        for (int q = 0; q < PER; q++) {
            pre[q] = run;
            run += x[q];
        }
        if (lane == 31) {
            sh.rowtot[warp] = incl & 0xffffu;
            sh.rowtot[warp + TC::kHalf] = incl >> 16;
        }
    }
    __syncthreads();  // (B)

    // ---- class runs (the scanning warps, lanes = classes): destination of
    // run c and its stage slot, at the destination's 16-byte phase within AU - 1
    // slots of slack per run; each scanning warp folds the slots into its row
    if (scans) {
        const uint32_t c = static_cast<uint32_t>(lane);
        const bool cls = c < static_cast<uint32_t>(M);
        const uint32_t cc = cls ? sh.rowtot[c] : 0u;
        const uint32_t cur = cls ? sh.cursor[par][c] : 0u;
        const uint32_t dst = FORWARD ? cur : cur - cc;
        const uint32_t room = cc + (cls ? AU - 1u : 0u);
        const uint32_t q0 = warp_incl_scan(room) - room;
        const uint32_t st = q0 + (((out.phase() + dst) - q0) & (AU - 1u));
        // slots < kStageElems < 2^16: the two classes' slots stay packed
        const uint32_t add = __shfl_sync(0xffffffffu, st, warp) |
                             (__shfl_sync(0xffffffffu, st, warp + TC::kHalf) << 16);
#pragma unroll
        for (int u = 0; u < PER / 4; u++)
            *reinterpret_cast<uint4*>(row + CC::chunk(lane, u)) =
                make_uint4(pre[4 * u] + add, pre[4 * u + 1] + add, pre[4 * u + 2] + add,
                           pre[4 * u + 3] + add);
        if (warp == 0 && cls) {
            sh.cursor[par ^ 1u][c] = FORWARD ? cur + cc : dst;
            sh.run_start[c] = st;
            sh.run_cnt[c] = cc;
            sh.run_dst[c] = run_position<OUT>(dst, st);
        }
    }
    // the stage is about to be rewritten: the previous tile's bulk stores
    // must have finished reading it
    if (tid < M) bulk_wait_read<0>();
    __syncthreads();  // (C)

    // ---- pass 2: scatter into the class-sorted stage
    auto place = [&](int j) {
        uint16_t& next = count_at(class_of(j));
        if constexpr (kRanks) {
            stage[next + ((lr[j >> 3] >> (4 * (j & 7))) & 15u)] = v[j];
        } else {  // the thread's slot of a class moves on with every element of it
            const uint32_t slot = next;
            next = static_cast<uint16_t>(slot + 1u);
            stage[slot] = v[j];
        }
    };
    if (CLUSTERED && one_class) {
        place_warp_run(stage + (count_at(c_last) - ITEMS * lane), v);
    } else if (full) {
#pragma unroll
        for (int j = 0; j < ITEMS; j++) place(j);
    } else {
#pragma unroll
        for (int j = 0; j < ITEMS; j++)
            if (e0 + j >= lo && e0 + j < hi) place(j);
    }
    fence_proxy_async_smem();
    __syncthreads();  // (D)

    if constexpr (!std::is_same<OUT, OutRows>::value) write_runs<V, M, THREADS>(stage, sh, out);
    return true;
}

// -------------------------------------------------------------- 2 classes --
// The filter case (m = 2; Haskell reference haskell_code/ParFilter.hs:8-21
// splits a list by a predicate, stably).  Same thread-contiguous elements
// and write-out as tile_scatter, with the counting done by bit masks:
//  * pass 1: each thread builds a mask of its class-1 elements (one bit per
//    element) and of its valid ones; its class counts are two popcounts; one
//    warp scan of the packed pair (class 0 low 16 bits, class 1 high) gives
//    each thread's prefix within the warp, lane 31 publishes the warp total;
//  * warp 0 scans the warp totals and places the two class runs at the
//    destination's 16-byte phase;
//  * pass 2: element j of a thread goes to its class's stage base + thread
//    prefix + popc(class mask & bits below j).
// No [class][thread] count matrix and no row scans: three barriers per tile
// instead of four and about half the instructions of the nibble step.  The
// scatter is bound by memory at m = 2 either way (N = 2^28 u32, B200: scatter
// kernel 0.383 ms with either step, against 0.337 ms for a plain 1 GiB
// device copy); the whole call at m = 2 is 1.02x the count kernel plus that
// copy.
template <class V, class D, int THREADS, bool FORWARD, class OUT, class AfterCounts, int ITEMS>
__device__ __forceinline__ bool tile_filter(const D& d, const V (&v)[ITEMS], uint32_t lo,
                                            uint32_t hi, bool full, V* stage, uint32_t* scr,
                                            TileShared<2>& sh, uint32_t par, const OUT& out, bool ok,
                                            AfterCounts after_counts) {
    using G = TileGeom<V, THREADS, 2, ITEMS * static_cast<int>(sizeof(V))>;
    constexpr uint32_t AU = OUT::kAU;
    constexpr int W = THREADS / 32;
    static_assert(ITEMS <= 16 && W <= 32, "16-bit packed warp counts, one lane per warp");
    uint32_t* wsum = scr;      // [W] packed class totals of each warp
    uint32_t* wpre = scr + W;  // [W] packed class prefixes of each warp

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t e0 = tid * ITEMS;

    // ---- pass 1: class-1 and valid masks, thread counts, warp prefixes
    uint32_t m1 = 0, mv = 0;
    if (full) {
#pragma unroll
        for (int j = 0; j < ITEMS; j++) m1 |= (d(v[j]) & 1u) << j;
        mv = (1u << ITEMS) - 1u;
    } else {
#pragma unroll
        for (int j = 0; j < ITEMS; j++) {
            if (e0 + j >= lo && e0 + j < hi) {
                m1 |= (d(v[j]) & 1u) << j;
                mv |= 1u << j;
            }
        }
    }
    const uint32_t n1 = static_cast<uint32_t>(__popc(m1));
    const bool one_class = full && warp_of_one_class(n1 == 0u || n1 == ITEMS, n1);
    const uint32_t x = (static_cast<uint32_t>(__popc(mv)) - n1) | (n1 << 16);
    const uint32_t incl = warp_incl_scan(x);
    if (lane == 31) wsum[warp] = incl;
    if (__syncthreads_or(!ok)) return false;  // (A)
    after_counts();

    // ---- the two class runs (warp 0; lane c = class c), warp prefixes
    if (warp == 0) {
        const uint32_t wt = lane < W ? wsum[lane] : 0u;
        const uint32_t wi = warp_incl_scan(wt);
        if (lane < W) wpre[lane] = wi - wt;
        const uint32_t tot = __shfl_sync(0xffffffffu, wi, 31);
        if (lane < 2) {
            const uint32_t c = static_cast<uint32_t>(lane);
            const uint32_t cc = c ? (tot >> 16) : (tot & 0xffffu);
            const uint32_t cur = sh.cursor[par][c];
            const uint32_t dst = FORWARD ? cur : cur - cc;
            const uint32_t q0 = c ? (tot & 0xffffu) + AU - 1u : 0u;  // class 0's room comes first
            const uint32_t st = q0 + (((out.phase() + dst) - q0) & (AU - 1u));
            sh.cursor[par ^ 1u][c] = FORWARD ? cur + cc : dst;
            sh.run_start[c] = st;
            sh.run_cnt[c] = cc;
            sh.run_dst[c] = run_position<OUT>(dst, st);
        }
    }
    // the stage is about to be rewritten: the previous tile's bulk stores
    // must have finished reading it
    if (tid < 2) bulk_wait_read<0>();
    __syncthreads();  // (B)

    // ---- pass 2: stage slot = class base + thread prefix + rank in the thread
    {
        const uint32_t pre = wpre[warp] + incl - x;
        const uint32_t b0 = sh.run_start[0] + (pre & 0xffffu);
        const uint32_t b1 = sh.run_start[1] + (pre >> 16);
        const uint32_t m0 = mv & ~m1;
        if (one_class) {
            place_warp_run(stage + ((m1 ? b1 : b0) - ITEMS * lane), v);
        } else {
#pragma unroll
            for (int j = 0; j < ITEMS; j++) {
                const uint32_t below = (1u << j) - 1u;
                const uint32_t slot = ((m1 >> j) & 1u)
                                          ? b1 + static_cast<uint32_t>(__popc(m1 & below))
                                          : b0 + static_cast<uint32_t>(__popc(m0 & below));
                if ((mv >> j) & 1u) stage[slot] = v[j];
            }
        }
    }
    fence_proxy_async_smem();
    __syncthreads();  // (C)

    if constexpr (!std::is_same<OUT, OutRows>::value) write_runs<V, 2, THREADS>(stage, sh, out);
    return true;
}

// ------------------------------------------------------------ 17..64 classes --
// With this many classes a thread's counters no longer fit in a register pair.
// They lie in shared memory instead, one byte per class, and are private to the
// thread, so no ranks have to be agreed on within a warp:
//  * pass 1: an element's local rank is the thread's counter of its class, read
//    and incremented.  A 32-bit word holds four classes, a row holds one word of
//    every thread, and a warp's 32 words of a row lie in 32 banks, so whatever
//    classes the lanes hold, a load or a store is one wavefront;
//  * scan: a warp takes a row (four classes), a lane the words of 8 or 16
//    threads; exclusive prefixes in the packed bytes, over as many lanes as keep
//    them within a byte (a group of 16 threads of 16 elements), are written back;
//    the lanes' totals, widened to 16 bits, are scanned over the warp and, with
//    the class's stage slot added, go to a [group][class] table;
//  * pass 2: stage slot = group table + thread prefix + local rank;
//  * the write-out is that of tile_scatter.
// The words lie in the columns of CountColumns; a row of the group table is
// padded by 8 bytes so that its 8-byte stores spread over the banks.
//
// What bounds it: the shared-memory pipe, about 15 wavefronts per 32 elements at
// m = 64 (a byte load and store, the two table lookups and the stage store of
// which the lookup and the store conflict at random), 70 % busy.  The ballots per
// class bit and shuffles that this replaces took 79 instructions an element and
// were bound by the ALU.  N = 2^28 u32, scatter at m = 32 and 64: 814 and 1050 us
// before, 528 and 707 with 256 threads, 506 and 597 with 512; 2^27 records of 8
// bytes: 521 and 632 before, 442 and 587, 443 and 501.
template <int M>
constexpr int kGroupRow = M + 4;  // u16 entries of a row of the group table

// Scan lanes (PER threads each) whose threads share a row of the group table:
// as many as keep a thread's prefix in the group within a byte, a warp at most.
__host__ __device__ constexpr int byte_group_lanes(int per, int items) {
    int l = 1;
    while (2 * l * per <= 32 && 2 * l * per * items <= 256) l *= 2;
    return l;
}

template <class V, class D, int M, int THREADS, bool FORWARD, bool CLUSTERED, class OUT,
          class AfterCounts, int ITEMS>
__device__ __forceinline__ bool tile_scatter_bytes(const D& d, const V (&v)[ITEMS], uint32_t lo,
                                                   uint32_t hi, bool full, V* stage,
                                                   unsigned char* cnt, TileShared<M>& sh,
                                                   uint32_t par, const OUT& out, bool ok,
                                                   AfterCounts after_counts) {
    using G = TileGeom<V, THREADS, M, ITEMS * static_cast<int>(sizeof(V))>;
    using CC = CountColumns<THREADS>;
    static_assert(G::kItems == ITEMS, "geometry");
    static_assert(M == 32 || M == 64, "class bound");
    constexpr uint32_t AU = OUT::kAU;
    constexpr int W = THREADS / 32;
    constexpr int PER = static_cast<int>(CC::kPer);
    constexpr int ROWS = M / 4;
    constexpr int RPW = (ROWS + W - 1) / W;  // rows a warp scans
    constexpr int LPG = byte_group_lanes(PER, ITEMS);
    static_assert((PER * LPG - 1) * ITEMS <= 255, "byte prefixes");
    static_assert(LPG == 1 || PER * ITEMS <= 255, "a lane's totals fit bytes when lanes share a group");

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t e0 = tid * ITEMS;
    unsigned char* my = cnt + 4u * CC::column(tid);  // class c at my[(c / 4) * 4 * THREADS + c % 4]
    uint16_t* grp = reinterpret_cast<uint16_t*>(cnt + M * THREADS);
    auto at = [&](uint32_t c) -> unsigned char& {
        return my[(c >> 2) * (4u * THREADS) + (c & 3u)];
    };

    // ---- pass 1: local ranks, a byte each
#pragma unroll
    for (int r = 0; r < ROWS; r++) *reinterpret_cast<uint32_t*>(my + r * 4 * THREADS) = 0u;
    uint32_t lr[(ITEMS + 3) / 4];
#pragma unroll
    for (int q = 0; q < (ITEMS + 3) / 4; q++) lr[q] = 0;
    constexpr bool kKeep = !CheapClass<D>::value;  // as in tile_scatter
    uint32_t kept[kKeep ? (ITEMS + 3) / 4 : 1];
    if constexpr (kKeep) {
#pragma unroll
        for (int q = 0; q < (ITEMS + 3) / 4; q++) kept[q] = 0;
    }
    auto class_of = [&](int j) -> uint32_t {
        if constexpr (kKeep) return __byte_perm(kept[j >> 2], 0u, 0x4440 + (j & 3));
        else return d(v[j]);
    };
    auto count = [&](int j) {
        const uint32_t c = d(v[j]);
        if constexpr (kKeep) kept[j >> 2] += c << (8 * (j & 3));
        unsigned char& x = at(c);
        const uint32_t r = x;
        x = static_cast<unsigned char>(r + 1u);
        lr[j >> 2] += r << (8 * (j & 3));
    };
    if (full) {
#pragma unroll
        for (int j = 0; j < ITEMS; j++) count(j);
    } else {
#pragma unroll
        for (int j = 0; j < ITEMS; j++)
            if (e0 + j >= lo && e0 + j < hi) count(j);
    }
    const uint32_t c_last = class_of(ITEMS - 1);
    bool one_class = false;  // the warp's elements
    if constexpr (CLUSTERED)
        one_class = full && warp_of_one_class(
                                (lr[(ITEMS - 1) >> 2] >> (8 * ((ITEMS - 1) & 3))) == ITEMS - 1, c_last);
    if (__syncthreads_or(!ok)) return false;  // (A)
    after_counts();

    // ---- scan: warp w takes rows w, w + W, ...; a lane PER threads
    uint32_t ev[RPW], od[RPW];  // classes 4 r, 4 r + 2 and 4 r + 1, 4 r + 3: exclusive over lanes
#pragma unroll
    for (int u = 0; u < RPW; u++) {
        const int r = warp + u * W;
        if (ROWS % W != 0 && r >= ROWS) break;
        unsigned char* row = cnt + 4 * r * THREADS;
        uint32_t x[PER];
#pragma unroll
        for (int q = 0; q < PER / 4; q++) {
            const uint4 a = *reinterpret_cast<const uint4*>(row + 4u * CC::chunk(lane, q));
            x[4 * q + 0] = a.x;
            x[4 * q + 1] = a.y;
            x[4 * q + 2] = a.z;
            x[4 * q + 3] = a.w;
        }
        uint32_t p = 0;  // the lane's threads but the last
#pragma unroll
        for (int q = 0; q + 1 < PER; q++) p += x[q];
        const uint32_t te = (p & 0x00ff00ffu) + (x[PER - 1] & 0x00ff00ffu);
        const uint32_t to = ((p >> 8) & 0x00ff00ffu) + ((x[PER - 1] >> 8) & 0x00ff00ffu);
        uint32_t run = 0;
        if constexpr (LPG > 1) {  // the threads of the group's lanes before this one
            const uint32_t own = p + x[PER - 1];
            uint32_t in = own;
#pragma unroll
            for (int dd = 1; dd < LPG; dd <<= 1) {
                const uint32_t up = __shfl_up_sync(0xffffffffu, in, dd, LPG);
                if (lane % LPG >= dd) in += up;
            }
            run = in - own;
        }
#pragma unroll
        for (int q = 0; q < PER; q++) {
            const uint32_t t = x[q];
            x[q] = run;
            run += t;
        }
#pragma unroll
        for (int q = 0; q < PER / 4; q++)
            *reinterpret_cast<uint4*>(row + 4u * CC::chunk(lane, q)) =
                make_uint4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
        const uint32_t ie = warp_incl_scan(te), io = warp_incl_scan(to);
        ev[u] = ie - te;
        od[u] = io - to;
        if (lane == 31) {
            *reinterpret_cast<uint4*>(&sh.rowtot[4 * r]) =
                make_uint4(ie & 0xffffu, io & 0xffffu, ie >> 16, io >> 16);
        }
    }
    __syncthreads();  // (B)

    // ---- class runs: destination of run c and its stage slot, at the
    // destination's 16-byte phase (every scanning warp, lanes = classes, two
    // consecutive classes a lane when M = 64)
    if (ROWS >= W || warp < ROWS) {
        constexpr int CPL = M > 32 ? 2 : 1;
        uint32_t cc[CPL], dst[CPL], st[CPL];
        uint32_t room = 0;
        const bool cls = lane * CPL < M;
#pragma unroll
        for (int q = 0; q < CPL; q++) {
            const int c = lane * CPL + q;
            cc[q] = cls ? sh.rowtot[c] : 0u;
            const uint32_t cur = cls ? sh.cursor[par][c] : 0u;
            dst[q] = FORWARD ? cur : cur - cc[q];
            room += cc[q] + (cls ? AU - 1u : 0u);
        }
        uint32_t q0 = warp_incl_scan(room) - room;
#pragma unroll
        for (int q = 0; q < CPL; q++) {
            st[q] = q0 + (((out.phase() + dst[q]) - q0) & (AU - 1u));
            q0 += cc[q] + AU - 1u;
        }
        if (warp == 0 && cls) {
#pragma unroll
            for (int q = 0; q < CPL; q++) {
                const int c = lane * CPL + q;
                sh.cursor[par ^ 1u][c] = FORWARD ? dst[q] + cc[q] : dst[q];
                sh.run_start[c] = st[q];
                sh.run_cnt[c] = cc[q];
                sh.run_dst[c] = run_position<OUT>(dst[q], st[q]);
            }
        }
        const uint32_t st2 = CPL == 2 ? st[0] | (st[CPL - 1] << 16) : st[0];  // slots < 2^16
#pragma unroll
        for (int u = 0; u < RPW; u++) {
            const int r = warp + u * W;
            if (ROWS % W != 0 && r >= ROWS) break;
            uint32_t s01, s23;  // the slots of classes 4 r, 4 r + 1 and 4 r + 2, 4 r + 3
            if (CPL == 2) {
                s01 = __shfl_sync(0xffffffffu, st2, 2 * r);
                s23 = __shfl_sync(0xffffffffu, st2, 2 * r + 1);
            } else {
                s01 = __shfl_sync(0xffffffffu, st2, 4 * r) |
                      (__shfl_sync(0xffffffffu, st2, 4 * r + 1) << 16);
                s23 = __shfl_sync(0xffffffffu, st2, 4 * r + 2) |
                      (__shfl_sync(0xffffffffu, st2, 4 * r + 3) << 16);
            }
            if (lane % LPG == 0)
                *reinterpret_cast<uint2*>(grp + (lane / LPG) * kGroupRow<M> + 4 * r) =
                    make_uint2(__byte_perm(ev[u], od[u], 0x5410) + s01,
                               __byte_perm(ev[u], od[u], 0x7632) + s23);
        }
    }
    // the stage is about to be rewritten: the previous tile's bulk stores
    // must have finished reading it
    if (tid < M) bulk_wait_read<0>();
    __syncthreads();  // (C)

    // ---- pass 2: scatter into the class-sorted stage
    const uint16_t* gb = grp + tid / (PER * LPG) * kGroupRow<M>;
    auto place = [&](int j) {
        const uint32_t c = class_of(j);
        stage[gb[c] + at(c) + __byte_perm(lr[j >> 2], 0u, 0x4440 + (j & 3))] = v[j];
    };
    if (CLUSTERED && one_class) {
        place_warp_run(stage + (gb[c_last] + at(c_last) - ITEMS * lane), v);
    } else if (full) {
        // Records whose neighbours share a class: stored in the threads' own order, lanes
        // of one class meet in two banks.  3 * 10^7 records of 8 bytes in runs of 300, a
        // call: m = 32 175 us without the look and 154 with it (256 threads), m = 64 200
        // and 167; the one-kernel form on sorted records, m = 32, 194 and 169.  Random
        // classes pay 1.8 and 0.3 % for the look.  4-byte values go without: their sixteen
        // a thread share a class less often, and in runs they were no slower than before.
        constexpr bool kSpread = !CLUSTERED && sizeof(V) >= 8;
        constexpr uint32_t kLast = 8 * ((ITEMS - 1) & 3);
        const bool one = kSpread && (lr[(ITEMS - 1) >> 2] >> kLast) == ITEMS - 1;
        const bool some = kSpread && __any_sync(0xffffffffu, one);
        if (some && one) {
#pragma unroll
            for (int q = 0; q < (ITEMS + 3) / 4; q++) lr[q] ^= spread_of<ITEMS>(lane) * 0x01010101u;
        }
#pragma unroll
        for (int j = 0; j < ITEMS; j++) place(j);
        if (some) order_lane_runs<V, ITEMS>(stage, one, gb[c_last] + at(c_last));
    } else {
#pragma unroll
        for (int j = 0; j < ITEMS; j++)
            if (e0 + j >= lo && e0 + j < hi) place(j);
    }
    fence_proxy_async_smem();
    __syncthreads();  // (D)

    if constexpr (!std::is_same<OUT, OutRows>::value) write_runs<V, M, THREADS>(stage, sh, out);
    return true;
}

}  // namespace mdx
