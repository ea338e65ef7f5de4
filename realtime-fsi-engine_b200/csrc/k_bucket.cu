// k_bucket.cu — predict, hash sort, cell table and reorder of a small scene
// (or batch) in four launches.
//
// The general path takes 13 launches a substep (predict, three radix passes of
// three, the table's clear and fill, the reorder), each a few microseconds of
// latency whatever its work: 35 us of a substep of 2,197 particles, and most
// of its launch time where no graph replays it.  Here the buckets are counted,
// the counts scanned, each particle id dropped into its bucket in order of
// arrival, and every slot then finds its id's rank among its bucket's ids,
// which is the order of the stable sort by (key, id), and gathers the particle
// there: 11 us.  Results are those of the general path, bit for bit.  (One
// cluster of eight blocks doing all but the last in one launch: 18 us for 2^17
// buckets and 67 for 1.5 * 2^20, eight SMs' worth of memory traffic.)
#include "pbf_batch.h"
#include "pbf_kernels.h"

namespace pbf {

constexpr int kScanThreads = 256;
constexpr uint32_t kScanOwn = 16, kScanTile = kScanThreads * kScanOwn;  // buckets a thread / a block scans
constexpr uint32_t kScanBlocks = kBucketSortMax / kScanTile;
static_assert(kScanBlocks <= 2 * kScanThreads, "the last block scans the block sums, two to a thread");

// Exclusive scan over the block's threads; *total: the block's sum.
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* s_warp, uint32_t* total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; ++w) {
        if (w == warp) before = all;
        all += s_warp[w];
    }
    *total = all;
    __syncthreads();
    return before + incl - v;
}

// keys and each particle's order of arrival in its bucket; cnt[buckets] is zero on entry.
template <bool B>
__global__ void __launch_bounds__(256) k_bucket_count(DevParams P, const SceneDev* __restrict__ scenes,
                                                      const uint16_t* __restrict__ scene_of,
                                                      const float4* __restrict__ pos, const float4* __restrict__ vel,
                                                      uint32_t* __restrict__ keys, uint32_t* __restrict__ arrival,
                                                      uint32_t* __restrict__ cnt)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    float3 vp, xs;
    predict_particle(P, __ldg(pos + i), __ldg(vel + i), vp, xs);
    uint32_t mask = P.mask, off = 0;
    if constexpr (B) {
        const SceneDev* S = scenes + __ldg(scene_of + i);
        mask = __ldg(&S->mask);
        off = __ldg(&S->table_off);
    }
    const uint32_t k = off + grid_hash(cell_coord(xs.x, P.h), cell_coord(xs.y, P.h), cell_coord(xs.z, P.h), mask);
    keys[i] = k;
    arrival[i] = atomicAdd(cnt + k, 1u);
}

// Starts of the buckets within their tile, and the tiles' starts (by the block
// that finishes last).  sums[kScanBlocks] counts the finished blocks, from 0.
__global__ void __launch_bounds__(kScanThreads) k_bucket_scan(uint32_t buckets, const uint32_t* __restrict__ cnt,
                                                              uint32_t* __restrict__ start, uint32_t* sums)
{
    __shared__ uint32_t s_warp[kScanThreads / 32];
    __shared__ bool s_last;
    const uint32_t at = (blockIdx.x * kScanThreads + threadIdx.x) * kScanOwn;
    uint32_t c[kScanOwn], mine = 0;
#pragma unroll
    for (uint32_t u = 0; u < kScanOwn; u += 4) {
        uint4 q = make_uint4(0, 0, 0, 0);
        if (at + u + 3 < buckets)
            q = __ldg(reinterpret_cast<const uint4*>(cnt + at + u));
        else if (at + u < buckets)  // (fewer than four buckets in all)
            q = make_uint4(__ldg(cnt + at + u), at + u + 1 < buckets ? __ldg(cnt + at + u + 1) : 0u,
                           at + u + 2 < buckets ? __ldg(cnt + at + u + 2) : 0u, 0u);
        c[u] = q.x;
        c[u + 1] = q.y;
        c[u + 2] = q.z;
        c[u + 3] = q.w;
    }
#pragma unroll
    for (uint32_t u = 0; u < kScanOwn; ++u) mine += c[u];
    uint32_t total;
    uint32_t s = block_scan(mine, s_warp, &total);
#pragma unroll
    for (uint32_t u = 0; u < kScanOwn; ++u) {
        if (c[u]) start[at + u] = s;
        s += c[u];
    }
    if (threadIdx.x == 0) {
        __stcg(sums + blockIdx.x, total);
        __threadfence();
        s_last = atomicAdd(sums + kScanBlocks, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const uint32_t b = threadIdx.x * 2u;
    const uint32_t v0 = b < gridDim.x ? __ldcg(sums + b) : 0u, v1 = b + 1u < gridDim.x ? __ldcg(sums + b + 1u) : 0u;
    const uint32_t before = block_scan(v0 + v1, s_warp, &total);
    if (b < gridDim.x) sums[b] = before;
    if (b + 1u < gridDim.x) sums[b + 1u] = before + v0;
    if (threadIdx.x == 0) sums[kScanBlocks] = 0u;
}

// The table, and the ids in their buckets in order of arrival.
__global__ void __launch_bounds__(256) k_bucket_place(uint32_t n, uint32_t buckets, const uint32_t* __restrict__ cnt,
                                                      const uint32_t* __restrict__ start,
                                                      const uint32_t* __restrict__ sums,
                                                      const uint32_t* __restrict__ keys,
                                                      const uint32_t* __restrict__ arrival, int2* __restrict__ table,
                                                      uint32_t* __restrict__ ids_in)
{
    const uint32_t stride = gridDim.x * blockDim.x, first = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t i = first; i < n; i += stride) {
        const uint32_t k = __ldg(keys + i);
        ids_in[__ldg(sums + k / kScanTile) + __ldg(start + k) + __ldg(arrival + i)] = i;
    }
    for (uint32_t k = first; k < buckets; k += stride) {
        const uint32_t c = __ldg(cnt + k);
        int2 se = make_int2(-1, -1);
        if (c) {
            const uint32_t s = __ldg(sums + k / kScanTile) + __ldg(start + k);
            se = make_int2((int)s, (int)(s + c));
        }
        table[k] = se;
    }
}

// Slot of id = ids_in[q]: its bucket's start plus the bucket's smaller ids.
// The gather is k_reorder's; cnt is left zero.
__global__ void __launch_bounds__(256) k_bucket_reorder(DevParams P, const uint32_t* __restrict__ ids_in,
                                                        uint32_t* __restrict__ cnt,
                                                        const uint32_t* __restrict__ keys,
                                                        const int2* __restrict__ table,
                                                        const float4* __restrict__ pos, const float4* __restrict__ vel,
                                                        uint32_t* __restrict__ ids, uint32_t* __restrict__ skeys,
                                                        float4* __restrict__ sx, float4* __restrict__ sv,
                                                        float4* __restrict__ sx0, uint32_t* __restrict__ lod)
{
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= P.n) return;
    const uint32_t id = __ldg(ids_in + q), key = __ldg(keys + id);
    const float4 p = __ldg(pos + id), v = __ldg(vel + id);
    const int2 se = __ldg(table + key);
    uint32_t s = (uint32_t)se.x;
    for (int x = se.x; x < se.y; ++x) s += __ldg(ids_in + x) < id ? 1u : 0u;
    ids[s] = id;
    if (skeys) skeys[s] = key;
    cnt[key] = 0u;
    reorder_particle(P, p, v, s, sx, sv, sx0, lod);
}

bool bucket_sort_fits(uint32_t n, uint32_t buckets) { return coop_lanes(n) != 0 && buckets <= kBucketSortMax; }

size_t bucket_scratch(uint32_t buckets) { return 2 * (size_t)((buckets + 3u) / 4u * 4u) + kScanBlocks + 1; }

void launch_bucket_sort(const DevParams& P, const SceneDev* scenes, const uint16_t* scene_of, const float4* pos,
                        const float4* vel, uint32_t* keys, uint32_t* arrival, uint32_t* scratch, uint32_t buckets,
                        int2* table, uint32_t* ids_in, uint32_t* ids, uint32_t* skeys, float4* sx, float4* sv, float4* sx0,
                        uint32_t* lod, int sms, cudaStream_t st, uint64_t* launches)
{
    uint32_t* cnt = scratch;
    uint32_t* start = cnt + (buckets + 3u) / 4u * 4u;
    uint32_t* sums = start + (buckets + 3u) / 4u * 4u;
    const unsigned g = (P.n + 255u) / 256u;
    if (scenes)
        k_bucket_count<true><<<g, 256, 0, st>>>(P, scenes, scene_of, pos, vel, keys, arrival, cnt);
    else
        k_bucket_count<false><<<g, 256, 0, st>>>(P, scenes, scene_of, pos, vel, keys, arrival, cnt);
    k_bucket_scan<<<(buckets + kScanTile - 1u) / kScanTile, kScanThreads, 0, st>>>(buckets, cnt, start, sums);
    const uint32_t most = buckets > P.n ? buckets : P.n, want = (most + 255u) / 256u, cap = (uint32_t)sms * 8u;
    k_bucket_place<<<want < cap ? want : cap, 256, 0, st>>>(P.n, buckets, cnt, start, sums, keys, arrival, table, ids_in);
    k_bucket_reorder<<<g, 256, 0, st>>>(P, ids_in, cnt, keys, table, pos, vel, ids, skeys, sx, sv, sx0, lod);
    *launches += 4;
}

}  // namespace pbf
