// mdx_small.cuh -- the plain stable partition of a few tiles as one launch.
//
// The CTAs of one thread-block cluster take a tile each, hold it in registers,
// exchange their class counts through distributed shared memory and place their
// elements by the plain scatter's tile step: one kernel that reads its input once,
// where the count and the scatter are two launches and read it twice.  What bounds
// it is latency: one round of loads, two cluster barriers and one tile step.  5003
// u32, m = 4: 14.2 us a call as two launches and 10.7 so, 8.2 and 5.8 replayed from a
// graph.
#pragma once

#include "mdx_device.cuh"
#include "mdx_plain.cuh"
#include "mdx_tile.cuh"

namespace mdx {

constexpr uint32_t kSmallTiles = 8;  // the portable cluster size

__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The u32 at `p` of this CTA's shared memory in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_load(const uint32_t* p, uint32_t rank) {
    uint32_t addr, v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(smem_addr(p)), "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

template <class V, int M, int THREADS>
struct SmallSmem {
    using G = TileGeom<V, THREADS, M>;
    static constexpr size_t kBytes = 128 + G::kStageBytes + G::kCntBytes;
};

// Grid = one cluster of num_tiles CTAs (at most kSmallTiles), tile b for CTA b.
template <class V, class D, int M, int THREADS>
__global__ void __launch_bounds__(THREADS) plain_small_kernel(PlainArgs a, D d, OutFlat<V> out) {
    using G = TileGeom<V, THREADS, M>;
    constexpr int ITEMS = G::kItems;
    constexpr int TILE = G::kTile;
    constexpr int W = THREADS / 32;
    constexpr uint32_t VE = 16 / sizeof(V);

    extern __shared__ __align__(128) unsigned char smem_raw[];
    const uint32_t raw = smem_addr(smem_raw);
    unsigned char* base = smem_raw + (((raw + 127u) & ~127u) - raw);
    V* stage = reinterpret_cast<V*>(base);
    uint32_t* cnt_sm = reinterpret_cast<uint32_t*>(base + G::kStageBytes);
    __shared__ TileShared<M> sh;
    __shared__ uint32_t own[M];     // this tile's class counts, read by the cluster
    __shared__ uint32_t red[W][M];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t k = blockIdx.x, tiles = gridDim.x;
    const uint64_t ts = static_cast<uint64_t>(k) * TILE;
    const uint32_t valid = static_cast<uint32_t>(min(static_cast<uint64_t>(TILE), a.n - ts));
    const bool full = valid == TILE;
    const uint32_t e0 = tid * ITEMS;
    const V* in = static_cast<const V*>(a.in) + ts;

    V v[ITEMS];
    if (full && (reinterpret_cast<uintptr_t>(in) & 15u) == 0) {
#pragma unroll
        for (uint32_t q = 0; q < ITEMS / VE; q++)
            unpack16_to<V>(__ldg(reinterpret_cast<const uint4*>(in + e0) + q), &v[q * VE]);
    } else {
#pragma unroll
        for (int j = 0; j < ITEMS; j++) v[j] = e0 + j < valid ? in[e0 + j] : V();
    }
    if (a.headflags != nullptr)
        for (uint32_t e = tid; e < valid; e += THREADS) a.headflags[ts + e] = 0u;

    // ---- the tile's class counts
    if constexpr (M <= 16) {
        PackedCounts<M> pc;
        pc.init();
#pragma unroll
        for (int j = 0; j < ITEMS; j++) {
            if (full || e0 + j < valid) pc.add(d(v[j]));
            if ((j & 7) == 7) pc.fold();
        }
        pc.finish();
#pragma unroll
        for (int c = 0; c < M; c++) {
            const uint32_t s = __reduce_add_sync(0xffffffffu, pc.acc[c]);
            if (lane == 0) red[warp][c] = s;
        }
    } else {
        for (int c = lane; c < M; c += 32) red[warp][c] = 0u;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < ITEMS; j++)
            if (full || e0 + j < valid) atomicAdd(&red[warp][d(v[j])], 1u);
    }
    __syncthreads();
    if (tid < M) {
        uint32_t s = 0;
#pragma unroll
        for (int w = 0; w < W; w++) s += red[w][tid];
        own[tid] = s;
    }
    cluster_arrive();
    cluster_wait();

    // ---- class bases and this tile's place in them (warp 0, lanes = classes)
    if (warp == 0) {
        uint32_t carry = 0;
#pragma unroll
        for (int h = 0; h < (M + 31) / 32; h++) {
            const int c = lane + 32 * h;
            uint32_t tot = 0, pre = 0;
            if (c < M) {
                for (uint32_t r = 0; r < tiles; r++) {
                    const uint32_t x = cluster_load(&own[c], r);
                    pre += r < k ? x : 0u;
                    tot += x;
                }
            }
            const uint32_t incl = warp_incl_scan(tot);
            const uint32_t bc = carry + incl - tot;
            if (c < M) {
                sh.cursor[0][c] = bc + pre;
                if (k == 0) {
                    a.class_base[c] = bc;
                    a.class_tot[c] = tot;
                    if (a.sizes != nullptr && static_cast<uint32_t>(c) < a.m) a.sizes[c] = tot;
                    // head-flag form (SeqMdiscr.h:47-49), zeroed before the cluster's barrier
                    if (a.headflags != nullptr && tot > 0) a.headflags[bc] = tot;
                }
            }
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    __syncthreads();
    cluster_arrive();  // this CTA has read the others' counts

    if constexpr (M == 2)
        (void)tile_filter<V, D, THREADS, true>(d, v, 0u, valid, full, stage, cnt_sm, sh, 0u, out, true, [] {});
    else if constexpr (M > 16)
        (void)tile_scatter_bytes<V, D, M, THREADS, true, true>(
            d, v, 0u, valid, full, stage, reinterpret_cast<unsigned char*>(cnt_sm), sh, 0u, out, true,
            [] {});
    else
        (void)tile_scatter<V, D, M, THREADS, true, true>(d, v, 0u, valid, full, stage, cnt_sm, sh, 0u,
                                                        out, true, [] {});
    if (tid < M) bulk_wait_all();
    cluster_wait();  // the others have read this one's
}

}  // namespace mdx
