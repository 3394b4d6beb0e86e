// mdx_wide.cu -- stable partition of wide elements: arrays of records of any
// width (the reference's _arrays variant, ModArray<N,LEN> over LEN u32 words,
// cuda_code/MdiscrHost_arrays.cu.h:26-36,250-430) and several columns that
// are permuted together (the _tuples variant's u32 / u8 / bool arrays,
// cuda_code/MdiscrHost_tuples.cu.h:13-48,262-429).
//
// Rows of up to kMaxRowBytes are moved whole through shared memory by the row
// kernels (mdx_rows.cuh).  Longer records go through 8-byte records:
//   1. build:     rec[i] = {key_i, i}        (key: the record's first u32 word)
//   2. partition: the REC8 kernels with the caller's discriminator on the key
//                 give the stable order of (key, row) and the class sizes;
//   3. gather:    output row p = input row (rec_out[p] >> 32).
// 4-, 8- and (16-byte aligned) 16-byte records take the element kernels.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "mdx_host.cuh"
#include "mdx_rows.cuh"

namespace mdx {
namespace wide {

constexpr int kThreads = 256;
// rec[i] = key_i | (i << 32), key_i = the u32 at byte offset stride * i of keys
__global__ void __launch_bounds__(kThreads) build_key_index(const unsigned char* keys, uint64_t stride,
                                                            uint64_t n, uint64_t* rec) {
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * kThreads + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * kThreads) {
        const uint32_t k = *reinterpret_cast<const uint32_t*>(keys + stride * i);
        rec[i] = static_cast<uint64_t>(k) | (i << 32);
    }
}

// Records of `words` u32 words: out row p = in row (perm[p] >> 32).  One
// thread per (row, word) pair, so a warp reads and writes consecutive words.
__global__ void __launch_bounds__(kThreads) gather_records(const uint32_t* in, uint32_t* out,
                                                           const uint64_t* perm, uint64_t n,
                                                           uint32_t words) {
    const uint64_t total = n * words;
    for (uint64_t t = static_cast<uint64_t>(blockIdx.x) * kThreads + threadIdx.x; t < total;
         t += static_cast<uint64_t>(gridDim.x) * kThreads) {
        const uint64_t p = t / words;
        const uint32_t w = static_cast<uint32_t>(t - p * words);
        const uint64_t src = perm[p] >> 32;
        out[t] = in[src * words + w];
    }
}

struct Layout {
    size_t rec_in, rec_out, plain, total;
    host::PlainLayout L;
};

// The REC8 partition's own workspace comes first, so its header (and the
// error word mdx_workspace_error reads) is the caller's; the two record
// arrays follow.
inline Layout layout(uint64_t n, uint32_t m) {
    Layout w;
    w.L = host::plain_layout(n, MDX_ELEM_REC8, m);
    w.plain = 0;
    w.rec_in = host::align_up(w.L.total, host::kAlign);
    w.rec_out = host::align_up(w.rec_in + 8 * n, host::kAlign);
    w.total = host::align_up(w.rec_out + 8 * n, host::kAlign);
    return w;
}

inline uint32_t grid_for(uint64_t work) {
    uint64_t g = (work + kThreads - 1) / kThreads;
    if (g > 148ull * 16) g = 148ull * 16;
    return static_cast<uint32_t>(g < 1 ? 1 : g);
}

// Steps 1-2: the stable order of (key, row) into rec_out, sizes and head flags.
inline mdx_status key_order(const unsigned char* keys, uint64_t stride, uint64_t n, mdx_discr discr,
                            uint32_t* d_sizes, uint32_t* d_headflags, unsigned char* ws,
                            const Layout& w, cudaStream_t st) {
    uint64_t* rec_in = reinterpret_cast<uint64_t*>(ws + w.rec_in);
    uint64_t* rec_out = reinterpret_cast<uint64_t*>(ws + w.rec_out);
    build_key_index<<<grid_for(n), kThreads, 0, st>>>(keys, stride, n, rec_in);
    if (cudaGetLastError() != cudaSuccess) return MDX_ERR_CUDA;
    return mdx_partition(rec_in, rec_out, n, MDX_ELEM_REC8, discr, d_sizes, d_headflags,
                         ws + w.plain, w.L.total, reinterpret_cast<mdx_stream_t>(st));
}

// The row kernels' tiles: 256 threads and two buffers of 20 KB, four CTAs to an SM
// (three at 9..16 classes with eight rows a thread: buffers of 18 KB, which make room
// for the fourth, were slower, 304 -> 315 us for 5 * 10^8 bytes of 20-byte rows); above
// 16 classes 512 threads and two of 36 KB, two CTAs, so that the byte counters' scan is
// shared by twice the rows (when it was taken, 2 * 10^7 rows of a key and 1, 2 and 8
// bytes, a call: m = 6 187 us with 256 threads, 192 with 512; m = 32 260 and 205).
constexpr int rows_threads(int M) { return M > 16 ? 512 : 256; }
constexpr uint32_t rows_buffer(int M) { return M > 32 ? 26624 : M > 16 ? 36864 : 20480; }
// At 33..64 classes the counters leave two CTAs 26 KB a buffer, enough for whole tiles
// (eight rows a thread) of rows of up to 6 bytes.  A tile of longer rows is cut by the
// buffer and pays for the same scan, so one CTA with two of 72 KB is better there.  A
// call at m = 64, one CTA with 36 KB (the only form before), two with 26 KB, one with
// 72 KB: 2 * 10^7 keys alone 198, 110, 198 us; with a column of 4 bytes 166, 152, 166
// (3 * 10^6: 26.8, 31.0, 26.8), with seven of one byte 314, 298, 250; 5 * 10^8 bytes of
// rows of 20 bytes 415, 369, 353, of 64 bytes 324, 303, 260, of 1000 bytes 386, 337, 200.
constexpr uint32_t kTwoCtaRowBytes = 6;
constexpr uint32_t rows_buffer(int M, uint32_t row_bytes) {
    return M > 32 && row_bytes > kTwoCtaRowBytes ? 73728 : rows_buffer(M);
}
constexpr int rows_ctas(int M, int items) { return M > 16 ? 2 : M > 8 && items == 8 ? 3 : 4; }
constexpr size_t kSmBytes = 228 * 1024;  // of an SM
constexpr size_t cta_bytes(int M) { return 1024 + 256 + 36 * M; }  // reserved, and the kernel's variables

// The row kernels take every record a tile of 16 of which fits the buffer and whose
// words do not outnumber the threads; the gathered route is behind at every width
// measured (6 * 10^8 bytes, m = 8: rows of 20, 64, 256 and 1024 bytes 929, 689, 559
// and 505 us gathered, 347, 317, 260 and 221 whole).
constexpr uint32_t kMaxRowBytes = 1024;
static_assert(16 * kMaxRowBytes + 16 <= rows_buffer(2) && kMaxRowBytes / 4 <= rows_threads(2), "tile of 16");

template <class D, int M, int ITEMS, bool RECORD>
mdx_status launch_rows(RowsArgs a, D d, uint32_t max_stride, cudaStream_t st) {
    constexpr int TS = rows_threads(M);
    auto scatter = rows_scatter_kernel<D, M, TS, ITEMS, RECORD>;
    using SL = RowsSmem<M, TS, ITEMS>;
    static_assert(rows_ctas(M, ITEMS) * (SL::bytes(rows_buffer(M)) + cta_bytes(M)) <= kSmBytes,
                  "CTAs of an SM");
    const size_t smem = SL::bytes(a.buf_bytes);
    // as many CTAs as the buffers leave room for: looked up for the two sizes they have
    // at most, not for each tile's own (short inputs have short tiles)
    const uint32_t most = a.buf_bytes <= rows_buffer(M) ? rows_buffer(M) : rows_buffer(M, kMaxRowBytes);
    int blocks = 0, sms = 0;
    if (host::occupancy(reinterpret_cast<const void*>(scatter), SL::bytes(most), &blocks, &sms, TS) !=
        cudaSuccess)
        return MDX_ERR_CUDA;
    uint32_t G = static_cast<uint32_t>(blocks) * static_cast<uint32_t>(sms);
    G = std::min(std::min(G, a.p.num_tiles), std::min(max_stride, host::kMaxChunks));
    a.p.num_chunks = G;
    a.p.chunk_stride = (G + 3u) & ~3u;
    if (a.p.headflags != nullptr &&
        cudaMemsetAsync(a.p.headflags, 0, a.p.n * sizeof(uint32_t), st) != cudaSuccess)
        return MDX_ERR_CUDA;
    rows_count_kernel<D, M><<<G, kRowsCountThreads, 0, st>>>(a, d);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(G);
    cfg.blockDim = dim3(TS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, scatter, a, d) != cudaSuccess) return MDX_ERR_CUDA;
    return cudaGetLastError() == cudaSuccess ? MDX_OK : MDX_ERR_CUDA;
}

template <class D, int M, bool RECORD>
mdx_status run_rows(RowsArgs a, D d, uint32_t max_stride, cudaStream_t st) {
    constexpr uint32_t TS = rows_threads(M);
    uint32_t row_bytes = 0;
    for (uint32_t c = 0; c < a.num_cols; c++) row_bytes += a.col[c].bytes;
    uint32_t room = rows_buffer(M, row_bytes);
    bool leads = false;
    for (uint32_t c = 0; c < a.num_cols; c++) {
        a.col[c].lead = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(a.col[c].in) % 16);
        if (a.col[c].lead != 0) {  // its tile takes a 16-byte word more
            leads = true;
            room -= 16;
        }
    }
    // eight rows a thread where that many (three quarters of them) fit the buffer,
    // else four; shorter tiles when that gives every SM two of them
    const uint32_t fit = room / row_bytes;
    const bool eight = fit >= 6 * TS;
    uint32_t T = std::min(fit & ~15u, TS * (eight ? 8u : 4u));
    while (T > 256 && a.p.n / T < 296) T = (T / 2) & ~15u;
    a.tile_rows = T;
    uint32_t off = 0;
    for (uint32_t c = 0; c < a.num_cols; c++) {
        RowsColumn& col = a.col[c];
        col.offset = off + col.lead;
        col.stride = T * col.bytes;  // T is a multiple of 16
        col.copied = (col.lead + col.stride + 15u) & ~15u;
        off += col.copied;
    }
    a.copied = off;
    a.key_offset = a.col[RECORD ? 0 : a.end[0]].offset;  // the first of the 4-byte columns
    a.buf_bytes = (off + 127u) & ~127u;
    a.p.num_tiles = static_cast<uint32_t>((a.p.n + T - 1) / T);
    // a copy of whole words ends up to 15 bytes past its tile: 16 rows of any column on
    a.bulk_tiles = static_cast<uint32_t>((a.p.n - (leads ? std::min<uint64_t>(a.p.n, 16) : 0)) / T);
    return eight ? launch_rows<D, M, 8, RECORD>(a, d, max_stride, st)
                 : launch_rows<D, M, 4, RECORD>(a, d, max_stride, st);
}

template <class D, bool RECORD>
mdx_status rows_by_bound(const RowsArgs& a, D d, uint32_t max_stride, cudaStream_t st) {
    switch (host::class_bound(a.p.m)) {
        case 2: return run_rows<D, 2, RECORD>(a, d, max_stride, st);
        case 4: return run_rows<D, 4, RECORD>(a, d, max_stride, st);
        case 8: return run_rows<D, 8, RECORD>(a, d, max_stride, st);
        case 16: return run_rows<D, 16, RECORD>(a, d, max_stride, st);
        case 32: return run_rows<D, 32, RECORD>(a, d, max_stride, st);
        default: return run_rows<D, 64, RECORD>(a, d, max_stride, st);
    }
}

// Rows held in a.col[0 .. num_cols); the keys are the first words of column 0.  The
// workspace is that of `layout`; the chunk counts may take the room of the record
// arrays, which the row kernels do not use.
template <bool RECORD>
mdx_status partition_rows(RowsArgs a, uint64_t n, mdx_discr discr, uint32_t* d_sizes,
                          uint32_t* d_headflags, unsigned char* ws, const Layout& w,
                          cudaStream_t st) {
    a.p = PlainArgs{};
    a.p.n = n;
    a.p.m = discr.m;
    a.p.chunk_cnt = reinterpret_cast<uint32_t*>(ws + w.L.chunk_cnt);
    a.p.class_base = reinterpret_cast<uint32_t*>(ws + w.L.class_base);
    a.p.class_tot = reinterpret_cast<uint32_t*>(ws + w.L.class_tot);
    a.p.sizes = d_sizes;
    a.p.headflags = d_headflags;
    a.p.error = &reinterpret_cast<host::WsHeader*>(ws)->error;
    a.p.prefix_in_scatter = 1;
    a.keys = a.col[0].in;
    a.key_stride = a.col[0].bytes;
    if (!RECORD) {  // the wider first; the key stays the first of its width
        std::stable_sort(a.col, a.col + a.num_cols,
                         [](const RowsColumn& x, const RowsColumn& y) { return x.bytes > y.bytes; });
        for (uint32_t q = 0; q < 4; q++)
            a.end[q] = static_cast<uint32_t>(
                std::count_if(a.col, a.col + a.num_cols,
                              [q](const RowsColumn& x) { return x.bytes >= (8u >> q); }));
    }
    const uint32_t M = host::class_bound(discr.m);
    const uint32_t max_stride = static_cast<uint32_t>(std::min<uint64_t>(
                                    (w.total - w.L.chunk_cnt) / (4ull * M), host::kMaxChunks)) & ~3u;
    if (host::use_mask(discr))
        return rows_by_bound<DiscrMask, RECORD>(a, DiscrMask{discr.m - 1u}, max_stride, st);
    return rows_by_bound<DiscrMod, RECORD>(a, DiscrMod::make(discr.m), max_stride, st);
}

}  // namespace wide
}  // namespace mdx

using namespace mdx;

extern "C" {

size_t mdx_records_workspace_size(uint64_t n, uint32_t record_bytes, uint32_t m) {
    if (record_bytes < 4 || record_bytes % 4 != 0 || m < 1 || m > MDX_MAX_CLASSES) return 0;
    if (record_bytes == 4) return mdx_workspace_size(n, MDX_ELEM_U32, m);
    if (record_bytes == 8) return mdx_workspace_size(n, MDX_ELEM_REC8, m);
    const size_t gathered = wide::layout(n, m).total;  // unaligned 16-byte records use it too
    if (record_bytes == 16) return std::max(gathered, mdx_workspace_size(n, MDX_ELEM_REC16, m));
    return gathered;
}

mdx_status mdx_partition_records(const void* d_in, void* d_out, uint64_t n, uint32_t record_bytes,
                                 mdx_discr discr, uint32_t* d_sizes, uint32_t* d_headflags,
                                 void* d_ws, size_t ws_bytes, mdx_stream_t stream) {
    if (record_bytes < 4 || record_bytes % 4 != 0) return MDX_ERR_INVALID;
    if (record_bytes == 4)
        return mdx_partition(d_in, d_out, n, MDX_ELEM_U32, discr, d_sizes, d_headflags, d_ws,
                             ws_bytes, stream);
    if (record_bytes == 8)
        return mdx_partition(d_in, d_out, n, MDX_ELEM_REC8, discr, d_sizes, d_headflags, d_ws,
                             ws_bytes, stream);
    if (record_bytes == 16 && reinterpret_cast<uintptr_t>(d_in) % 16 == 0 &&
        reinterpret_cast<uintptr_t>(d_out) % 16 == 0)  // the 16-byte record kernels
        return mdx_partition(d_in, d_out, n, MDX_ELEM_REC16, discr, d_sizes, d_headflags, d_ws,
                             ws_bytes, stream);
    mdx_status s = host::check_discr(discr);
    if (s != MDX_OK) return s;
    if (n > MDX_MAX_ELEMS) return MDX_ERR_INVALID;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (n == 0) {
        if (d_sizes && cudaMemsetAsync(d_sizes, 0, discr.m * sizeof(uint32_t), st) != cudaSuccess)
            return MDX_ERR_CUDA;
        return MDX_OK;
    }
    if (d_in == nullptr || d_out == nullptr) return MDX_ERR_INVALID;
    if (reinterpret_cast<uintptr_t>(d_in) % 4 || reinterpret_cast<uintptr_t>(d_out) % 4)
        return MDX_ERR_INVALID;
    const char* ib = static_cast<const char*>(d_in);
    const char* ob = static_cast<const char*>(d_out);
    if (ib < ob + n * record_bytes && ob < ib + n * record_bytes) return MDX_ERR_INVALID;
    const wide::Layout w = wide::layout(n, discr.m);
    if (d_ws == nullptr || ws_bytes < w.total || reinterpret_cast<uintptr_t>(d_ws) % host::kAlign)
        return MDX_ERR_WORKSPACE;
    unsigned char* ws = static_cast<unsigned char*>(d_ws);
    if (record_bytes <= wide::kMaxRowBytes) {
        RowsArgs a{};
        a.num_cols = 1;
        RowsColumn& c = a.col[0];
        c.in = static_cast<const unsigned char*>(d_in);
        c.out = static_cast<unsigned char*>(d_out);
        c.bytes = record_bytes;
        c.unit = 16;
        while (record_bytes % c.unit || reinterpret_cast<uintptr_t>(d_in) % c.unit ||
               reinterpret_cast<uintptr_t>(d_out) % c.unit)
            c.unit /= 2;  // 4 divides all three
        return wide::partition_rows<true>(a, n, discr, d_sizes, d_headflags, ws, w, st);
    }
    s = wide::key_order(static_cast<const unsigned char*>(d_in), record_bytes, n, discr, d_sizes,
                        d_headflags, ws, w, st);
    if (s != MDX_OK) return s;
    const uint32_t words = record_bytes / 4;
    wide::gather_records<<<wide::grid_for(n * words), wide::kThreads, 0, st>>>(
        static_cast<const uint32_t*>(d_in), static_cast<uint32_t*>(d_out),
        reinterpret_cast<const uint64_t*>(ws + w.rec_out), n, words);
    return cudaGetLastError() == cudaSuccess ? MDX_OK : MDX_ERR_CUDA;
}

size_t mdx_columns_workspace_size(uint64_t n, uint32_t m) {
    if (m < 1 || m > MDX_MAX_CLASSES) return 0;
    return wide::layout(n, m).total;
}

mdx_status mdx_partition_columns(const mdx_column* cols, uint32_t num_cols, uint64_t n,
                                 mdx_discr discr, uint32_t* d_sizes, uint32_t* d_headflags,
                                 void* d_ws, size_t ws_bytes, mdx_stream_t stream) {
    if (cols == nullptr || num_cols < 1 || num_cols > static_cast<uint32_t>(kMaxCols))
        return MDX_ERR_INVALID;
    mdx_status s = host::check_discr(discr);
    if (s != MDX_OK) return s;
    if (n > MDX_MAX_ELEMS || cols[0].elem_bytes != 4) return MDX_ERR_INVALID;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (n == 0) {
        if (d_sizes && cudaMemsetAsync(d_sizes, 0, discr.m * sizeof(uint32_t), st) != cudaSuccess)
            return MDX_ERR_CUDA;
        return MDX_OK;
    }
    RowsArgs a{};
    a.num_cols = num_cols;
    for (uint32_t i = 0; i < num_cols; i++) {
        const uint32_t b = cols[i].elem_bytes;
        if ((b != 1 && b != 2 && b != 4 && b != 8) || cols[i].in == nullptr || cols[i].out == nullptr ||
            reinterpret_cast<uintptr_t>(cols[i].in) % b || reinterpret_cast<uintptr_t>(cols[i].out) % b)
            return MDX_ERR_INVALID;
        for (uint32_t j = 0; j < num_cols; j++) {  // no output may overlap any input or output
            const char* o = static_cast<const char*>(cols[i].out);
            const char* x = static_cast<const char*>(cols[j].in);
            if (o < x + n * cols[j].elem_bytes && x < o + n * b) return MDX_ERR_INVALID;
            if (j != i) {
                const char* y = static_cast<const char*>(cols[j].out);
                if (o < y + n * cols[j].elem_bytes && y < o + n * b) return MDX_ERR_INVALID;
            }
        }
        a.col[i].in = static_cast<const unsigned char*>(cols[i].in);
        a.col[i].out = static_cast<unsigned char*>(cols[i].out);
        a.col[i].bytes = b;
        a.col[i].unit = b;
    }
    const wide::Layout w = wide::layout(n, discr.m);
    if (d_ws == nullptr || ws_bytes < w.total || reinterpret_cast<uintptr_t>(d_ws) % host::kAlign)
        return MDX_ERR_WORKSPACE;
    return wide::partition_rows<false>(a, n, discr, d_sizes, d_headflags,
                                       static_cast<unsigned char*>(d_ws), w, st);
}

}  // extern "C"
