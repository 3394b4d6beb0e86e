// mdx_rows.cuh -- stable partition of rows that are not one 4-, 8- or 16-byte
// element: records of any multiple of 4 bytes, and several columns that are
// permuted together.
//
//   rows_count_kernel    the class counts of every chunk of row tiles, from the
//                        keys alone;
//   rows_scatter_kernel  CTA k walks chunk k from its end.  A tile's rows come into
//                        shared memory whole (one bulk copy per column, the next
//                        tile's while this one is placed); the tile step of the
//                        plain scatter ranks {class, row} words, which leaves the
//                        tile's row numbers in class order in the stage; the rows
//                        are then stored from there, consecutive words of the
//                        output by consecutive threads.
//
// Rows are read once for their keys and once to be moved, and written once,
// without intermediates.  The {key, row} records, partitioned as 8-byte elements
// and followed by a gather of the rows, that this replaces cost 48 bytes of
// traffic a row beyond that, and the gather's reads touched every sector once for
// each class.  3 * 10^7 rows of 20 bytes, m = 8: 924 -> 345 us a call (scatter about
// 235, count 108; read twice and written once at the copy rate: 275).  2 * 10^7 rows of
// a key and columns of 1, 2 and 8 bytes, m = 6: 415 -> 148 us (floor 104).  Rows of
// 32 bytes and more are bound by memory, narrower ones by the instructions a row
// costs (ranks, two table lookups, a load and a store per column).
#pragma once

#include "mdx_device.cuh"
#include "mdx_plain.cuh"
#include "mdx_tile.cuh"

namespace mdx {

constexpr int kMaxCols = 8;
constexpr int kRowsCountThreads = 256;

struct RowsColumn {
    const unsigned char* in;
    unsigned char* out;
    uint32_t bytes;   // of a row
    uint32_t unit;    // 1, 2, 4, 8 or 16: bytes moved at a time
    uint32_t offset;  // of the column's tile in a tile buffer
    uint32_t lead;    // bytes of the column's first 16-byte word before its first row
    uint32_t copied;  // bytes of the 16-byte words that hold a whole tile
    uint32_t stride;  // bytes of a whole tile
};

struct RowsArgs {
    PlainArgs p;          // n, num_tiles, chunks and counts, sizes, head flags, error (in, out unused)
    const unsigned char* keys;
    uint32_t key_stride;  // bytes between keys
    uint32_t tile_rows;   // rows of a tile, a multiple of 16
    uint32_t buf_bytes;   // of a tile buffer
    uint32_t copied;      // bytes that a whole tile's copies bring
    uint32_t key_offset;  // of the key column's tile in a tile buffer
    uint32_t num_cols;
    uint32_t bulk_tiles;  // whole tiles that come by bulk copies: all of them, but when a
                          // column has a lead not the last (its copy could pass the end)
    uint32_t end[4];      // columns (not a record): end[q] of 8 >> q bytes or more, the wider first
    RowsColumn col[kMaxCols];
};

// The tile step's elements: a row's number in the tile and its class above it.
struct DiscrRow {
    __device__ __forceinline__ uint32_t operator()(uint32_t v) const { return v >> 16; }
};

template <>
struct CheapClass<DiscrRow> : std::true_type {};

template <class D, int M>
__global__ void __launch_bounds__(kRowsCountThreads, 4) rows_count_kernel(const __grid_constant__ RowsArgs a, D d) {
    constexpr int W = kRowsCountThreads / 32;
    constexpr int U = 8;
    __shared__ uint32_t red[W][M];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, k = blockIdx.x;
    pdl_launch_dependents();
    uint32_t t0, t1;
    chunk_tiles(k, a.p.num_tiles, a.p.num_chunks, t0, t1);
    const uint64_t r0 = static_cast<uint64_t>(t0) * a.tile_rows;
    const uint64_t r1 = min(static_cast<uint64_t>(t1) * a.tile_rows, a.p.n);
    auto key = [&](uint64_t r) {
        return __ldg(reinterpret_cast<const uint32_t*>(a.keys + r * a.key_stride));
    };
    PackedCounts<M <= 16 ? M : 16> pc;
    pc.init();
    auto count = [&](uint32_t x) {
        if constexpr (M <= 16) pc.add(d(x));
        else atomicAdd(&red[warp][d(x)], 1u);
    };
    for (uint32_t c = lane; c < M; c += 32) red[warp][c] = 0u;
    __syncwarp();
    uint64_t first = r0;  // rows that the 16-byte loads do not take
    if (a.key_stride == 4u && (reinterpret_cast<uintptr_t>(a.keys) & 15u) == 0) {
        const uint4* kv = reinterpret_cast<const uint4*>(a.keys + 4u * r0);  // r0: a multiple of 16
        const uint64_t nv = (r1 - r0) / 4u;
        constexpr int UV = 4;
        for (uint64_t i = tid; i < nv; i += UV * kRowsCountThreads) {
            uint4 x[UV];
#pragma unroll
            for (int u = 0; u < UV; u++)
                if (i + u * kRowsCountThreads < nv) x[u] = __ldg(kv + i + u * kRowsCountThreads);
#pragma unroll
            for (int u = 0; u < UV; u++) {
                if (i + u * kRowsCountThreads < nv) {
                    count(x[u].x);
                    count(x[u].y);
                    count(x[u].z);
                    count(x[u].w);
                }
                if constexpr (M <= 16)
                    if (u & 1) pc.fold();  // every 8 increments
            }
        }
        first = r0 + 4u * nv;
    }
    for (uint64_t r = first + tid; r < r1; r += U * kRowsCountThreads) {
        uint32_t x[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (r + u * kRowsCountThreads < r1) x[u] = key(r + u * kRowsCountThreads);
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (r + u * kRowsCountThreads < r1) count(x[u]);
        }
        if constexpr (M <= 16) pc.fold();  // every 8 increments
    }
    if constexpr (M <= 16) {
        pc.finish();
#pragma unroll
        for (int c = 0; c < M; c++) {
            const uint32_t s = warp_sum(pc.acc[c]);
            if (lane == 0) red[warp][c] = s;
        }
    }
    __syncthreads();
    if (tid < M) {
        uint32_t s = 0;
#pragma unroll
        for (int w = 0; w < W; w++) s += red[w][tid];
        a.p.chunk_cnt[static_cast<uint64_t>(tid) * a.p.chunk_stride + k] = s;
    }
}

template <int M, int THREADS, int ITEMS>
struct RowsSmem {
    using G = TileGeom<uint32_t, THREADS, M, ITEMS * 4>;
    static constexpr int kRows = THREADS * ITEMS;  // rows of a tile at most
    static constexpr size_t kStage = G::kStageBytes, kCnt = (G::kCntBytes + 15) / 16 * 16;
    static constexpr size_t bytes(size_t buf_bytes) {
        return 128 + 2 * buf_bytes + kStage + kCnt + kRows;
    }
};

// How the threads share the words of a record tile: consecutive threads take
// consecutive words of consecutive slots, a thread keeps its word (the threads past
// the last whole row of words rest).
struct RowShare {
    uint32_t first, step, word;
};

// The tile's rows in their order: slot s takes row stage[s] in shared memory to row
// s + run_dst[class] of the output.
template <class T, int M>
__device__ __forceinline__ void write_records(const RowsColumn& col, const unsigned char* tile,
                                              const uint32_t* stage, const TileShared<M>& sh,
                                              uint32_t rows, const RowShare& share) {
    const uint32_t bytes = col.bytes, at = share.word * static_cast<uint32_t>(sizeof(T));
    const unsigned char* src = tile + col.offset + at;
    unsigned char* out = col.out + at;
#pragma unroll 4
    for (uint32_t s = share.first; s < rows; s += share.step) {
        const uint32_t x = stage[s];
        const T val = *reinterpret_cast<const T*>(src + (x & 0xffffu) * bytes);
        const uint32_t row = s + sh.run_dst[x >> 16];
        *reinterpret_cast<T*>(out + static_cast<uint64_t>(row) * bytes) = val;
    }
}

// The same for columns, all of a slot's at once, N slots a thread, the columns in
// order of their widths: a.end[q] columns of 8 >> q bytes or more.  ALL: the N slots
// are there; otherwise the thread's first is, and the others if below `rows`.
template <class T, int N, bool ALL>
__device__ __forceinline__ void move_column(const RowsColumn& col, const unsigned char* tile,
                                            const uint32_t (&from)[N], const uint32_t (&to)[N],
                                            uint32_t slots) {
    const T* src = reinterpret_cast<const T*>(tile + col.offset);
    T* out = reinterpret_cast<T*>(col.out);
    T val[N];
#pragma unroll
    for (int q = 0; q < N; q++) val[q] = src[from[q]];
#pragma unroll
    for (int q = 0; q < N; q++)
        if (ALL || static_cast<uint32_t>(q) < slots) out[to[q]] = val[q];
}
template <int M, int THREADS, int N, bool ALL>
__device__ __forceinline__ void move_slots(const RowsArgs& a, const unsigned char* tile,
                                           const uint32_t* stage, const TileShared<M>& sh,
                                           uint32_t s, uint32_t rows) {
    const uint32_t slots = ALL ? N : min(static_cast<uint32_t>(N), (rows - s + THREADS - 1u) / THREADS);
    uint32_t from[N], to[N];
#pragma unroll
    for (int q = 0; q < N; q++) {
        const uint32_t sl = ALL || static_cast<uint32_t>(q) < slots ? s + q * THREADS : s;
        const uint32_t x = stage[sl];
        from[q] = x & 0xffffu;
        to[q] = sl + sh.run_dst[x >> 16];
    }
    uint32_t c = 0;
    for (; c < a.end[0]; c++) move_column<uint64_t, N, ALL>(a.col[c], tile, from, to, slots);
    for (; c < a.end[1]; c++) move_column<uint32_t, N, ALL>(a.col[c], tile, from, to, slots);
    for (; c < a.end[2]; c++) move_column<uint16_t, N, ALL>(a.col[c], tile, from, to, slots);
    for (; c < a.end[3]; c++) move_column<uint8_t, N, ALL>(a.col[c], tile, from, to, slots);
}
template <int M, int THREADS>
__device__ __forceinline__ void write_columns(const RowsArgs& a, const unsigned char* tile,
                                              const uint32_t* stage, const TileShared<M>& sh,
                                              uint32_t rows) {
    uint32_t base = 0;
    for (; base + 4 * THREADS <= rows; base += 4 * THREADS)
        move_slots<M, THREADS, 4, true>(a, tile, stage, sh, base + threadIdx.x, rows);
    for (uint32_t s = base + threadIdx.x; s < rows; s += 2 * THREADS)
        move_slots<M, THREADS, 2, false>(a, tile, stage, sh, s, rows);
}

template <class T, int THREADS>
__device__ __forceinline__ void load_rows(const RowsColumn& col, unsigned char* tile, uint64_t row0,
                                          uint32_t rows) {
    const uint32_t W = col.bytes / sizeof(T);
    const T* src = reinterpret_cast<const T*>(col.in) + row0 * W;
    T* dst = reinterpret_cast<T*>(tile + col.offset);
    for (uint32_t o = threadIdx.x; o < rows * W; o += THREADS) dst[o] = src[o];
}

template <class D, int M, int THREADS, int ITEMS, bool RECORD>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS)
    rows_scatter_kernel(const __grid_constant__ RowsArgs a, D d) {
    using L = RowsSmem<M, THREADS, ITEMS>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const uint32_t raw = smem_addr(smem_raw);
    unsigned char* base = smem_raw + (((raw + 127u) & ~127u) - raw);
    unsigned char* bufs = base;
    uint32_t* stage = reinterpret_cast<uint32_t*>(base + 2 * static_cast<size_t>(a.buf_bytes));
    uint32_t* cnt_sm = stage + L::kStage / 4;
    unsigned char* cls = reinterpret_cast<unsigned char*>(cnt_sm) + L::kCnt;  // class of each row

    __shared__ __align__(8) uint64_t bars[2];
    __shared__ TileShared<M> sh;
    __shared__ uint32_t tot_sh[M], pre_sh[M];
    __shared__ int clustered_sh;

    const uint32_t tid = threadIdx.x;
    const uint32_t k = blockIdx.x, T = a.tile_rows;
    uint32_t t0, t1;
    chunk_tiles(k, a.p.num_tiles, a.p.num_chunks, t0, t1);
    const uint32_t cnt = t1 - t0;
    if (cnt == 0) return;
    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        mbar_fence_init();
    }
    if (tid < M) {
        tot_sh[tid] = 0u;
        pre_sh[tid] = 0u;
    }
    __syncthreads();

    // i-th tile in processing order is tile t1-1-i.  A tile's rows come by one bulk copy
    // per column, of the 16-byte words that hold them: a column off a 16-byte address
    // lies `lead` bytes into its room.  Element loads with a barrier after them, which
    // took the place of the copies there: 5 * 10^8 bytes at 4 bytes off, a call, rows of
    // 20 bytes m = 8 412 us, now 274 (aligned 271), of 256 bytes 363 and 226 (212: its
    // rows move by 4 bytes, not 16); 2 * 10^7 rows of a key and seven columns of 8 bytes,
    // m = 2, 1093 and 452 (446).
    auto rows_of = [&](uint32_t tile) {
        return static_cast<uint32_t>(
            min(static_cast<uint64_t>(T), a.p.n - static_cast<uint64_t>(tile) * T));
    };
    auto issue = [&](uint32_t i) {  // thread 0: the columns of tile i
        const uint32_t tile = t1 - 1u - i;
        uint64_t* bar = &bars[i & 1u];
        unsigned char* buf = bufs + (i & 1u) * static_cast<size_t>(a.buf_bytes);
        if (tile >= a.bulk_tiles) {
            mbar_arrive(bar);
            return;
        }
        mbar_arrive_expect_tx(bar, a.copied);
        for (uint32_t c = 0; c < (RECORD ? 1u : a.num_cols); c++) {
            const RowsColumn& col = a.col[c];
            bulk_load_g2s(buf + col.offset - col.lead,
                          col.in - col.lead + static_cast<uint64_t>(tile) * col.stride, col.copied, bar);
        }
    };
    if (tid == 0) issue(0);
    RowShare share{0u, 1u, 0u};
    if constexpr (RECORD) {
        const uint32_t W = a.col[0].bytes / a.col[0].unit;
        const uint32_t whole = THREADS / W;  // rows of words the threads hold at once
        share = RowShare{tid < whole * W ? tid / W : 0xffffffffu, whole, tid % W};
    }
    pdl_wait();
    scatter_cursors<M, THREADS>(a.p, k, tot_sh, pre_sh, sh.cursor[0], &clustered_sh);
    __syncthreads();

    for (uint32_t i = 0; i < cnt; i++) {
        const uint32_t tile = t1 - 1u - i;
        const uint32_t rows = rows_of(tile);
        unsigned char* buf = bufs + (i & 1u) * static_cast<size_t>(a.buf_bytes);
        const bool ok = mbar_wait_bounded(&bars[i & 1u], (i >> 1) & 1u);
        if (tile >= a.bulk_tiles) {  // no bulk copy brought it
            for (uint32_t c = 0; c < a.num_cols; c++) {
                const uint64_t row0 = static_cast<uint64_t>(tile) * T;
                if constexpr (RECORD) {
                    load_rows<uint32_t, THREADS>(a.col[c], buf, row0, rows);
                } else {
                    switch (a.col[c].bytes) {
                        case 1: load_rows<uint8_t, THREADS>(a.col[c], buf, row0, rows); break;
                        case 2: load_rows<uint16_t, THREADS>(a.col[c], buf, row0, rows); break;
                        case 4: load_rows<uint32_t, THREADS>(a.col[c], buf, row0, rows); break;
                        default: load_rows<uint64_t, THREADS>(a.col[c], buf, row0, rows); break;
                    }
                }
            }
            __syncthreads();
        }
        uint32_t v[ITEMS];
        const uint32_t e0 = tid * ITEMS;
        if constexpr (RECORD) {
            // a row's class by the thread that meets the fewest bank conflicts on the
            // keys, to the thread that ranks it
            for (uint32_t r = tid; r < rows; r += THREADS)
                cls[r] = static_cast<unsigned char>(
                    ok ? d(*reinterpret_cast<const uint32_t*>(buf + a.key_offset + r * a.key_stride)) : 0u);
            __syncthreads();
#pragma unroll
            for (int q = 0; q < ITEMS / 4; q++) {
                const uint32_t x = reinterpret_cast<const uint32_t*>(cls + e0)[q];
#pragma unroll
                for (int j = 0; j < 4; j++) v[4 * q + j] = (e0 + 4 * q + j) | (((x >> (8 * j)) & 0xffu) << 16);
            }
        } else {  // a column of keys: the thread's own, in 16-byte words
            const uint32_t off = (a.key_offset >> 2) & 3u;  // keys before the thread's in its first
            const uint4* keys = reinterpret_cast<const uint4*>(buf + a.key_offset - 4u * off + 4u * e0);
            const uint4 none = make_uint4(0u, 0u, 0u, 0u);
            if (off == 0u) {  // the same for every thread of the grid
#pragma unroll
                for (int q = 0; q < ITEMS / 4; q++) {
                    const uint4 x = ok && e0 + 4 * q < rows ? keys[q] : none;
                    const uint32_t r = e0 + 4 * q;
                    v[4 * q] = r | (d(x.x) << 16);
                    v[4 * q + 1] = (r + 1) | (d(x.y) << 16);
                    v[4 * q + 2] = (r + 2) | (d(x.z) << 16);
                    v[4 * q + 3] = (r + 3) | (d(x.w) << 16);
                }
            } else {
                uint32_t x[ITEMS + 4];
#pragma unroll
                for (int q = 0; q <= ITEMS / 4; q++) {
                    const uint4 k = ok && e0 + 4 * q < rows + off ? keys[q] : none;
                    x[4 * q] = k.x;
                    x[4 * q + 1] = k.y;
                    x[4 * q + 2] = k.z;
                    x[4 * q + 3] = k.w;
                }
#pragma unroll
                for (int j = 0; j < ITEMS; j++)
                    v[j] = (e0 + j) |
                           (d(off == 1u ? x[j + 1] : off == 2u ? x[j + 2] : x[j + 3]) << 16);
            }
        }
        auto next = [&] {  // every thread has stored the rows of the other buffer
            if (tid == 0 && i + 1 < cnt) issue(i + 1);
        };
        const bool full = rows == static_cast<uint32_t>(L::kRows);
        bool done;
        if constexpr (M == 2)
            done = tile_filter<uint32_t, DiscrRow, THREADS, false>(
                DiscrRow{}, v, 0u, rows, full, stage, cnt_sm, sh, i & 1u, OutRows{}, ok, next);
        else if constexpr (M > 16)
            done = tile_scatter_bytes<uint32_t, DiscrRow, M, THREADS, false, false>(
                DiscrRow{}, v, 0u, rows, full, stage, reinterpret_cast<unsigned char*>(cnt_sm), sh,
                i & 1u, OutRows{}, ok, next);
        else
            done = tile_scatter<uint32_t, DiscrRow, M, THREADS, false, false>(
                DiscrRow{}, v, 0u, rows, full, stage, cnt_sm, sh, i & 1u, OutRows{}, ok, next);
        if (!done) {  // nothing of this tile written; no later copy is in flight
            if (tid == 0) {
                atomicOr(a.p.error, kErrTimeout);
                (void)mbar_wait_bounded(&bars[i & 1u], (i >> 1) & 1u);
            }
            break;
        }
        if constexpr (RECORD) {
            switch (a.col[0].unit) {
                case 4: write_records<uint32_t, M>(a.col[0], buf, stage, sh, rows, share); break;
                case 8: write_records<uint64_t, M>(a.col[0], buf, stage, sh, rows, share); break;
                default: write_records<uint4, M>(a.col[0], buf, stage, sh, rows, share); break;
            }
        } else {
            write_columns<M, THREADS>(a, buf, stage, sh, rows);
        }
        // this buffer's generic accesses precede the copy that refills it
        fence_proxy_async_smem();
    }
}

}  // namespace mdx
