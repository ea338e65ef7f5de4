// coop_walk.cuh — the walk of a particle's 27 hashed buckets by a group of G
// lanes, shared by the passes of k_coop.cu and their adjoints (k_adjoint.cu).
#pragma once

#include <utility>

#include "masked_body.cuh"
#include "pbf_kernels.h"

namespace pbf {

constexpr int kCThreads = 128;
// 8 resident blocks (64 registers): the lists of a block take 13-16 KB of the
// SM's 256 KB of shared memory and L1, and what is left over caches the
// neighbours' positions, so more residency does not pay (a lambda pass of
// 32,768 particles at G = 8: 22.4 us; 6 blocks: 23.0, 10: 24.7, 12: 29.3).
constexpr int kCBlocks = 8;

// The passes over kept hits: loads of 4 chunks of G hits in flight, 8 resident
// blocks (131,072 particles, delta-p / reverse delta-p / reverse lambda: 22.5 /
// 31.6 / 24.2 us; 2 chunks 23.4 / 31.9 / 24.7, 8 chunks 22.1 / 34.8 / 24.4; 12
// blocks of 2 chunks 23.3 / 38.0 / 24.0, 16 of 1 chunk 26.4 / 49.9 / 23.4: the
// obstacle's reverse projection spills).
constexpr int kReplayAhead = 4, kReplayBlocks = 8;

template <int G>
struct CoopShape {
    static constexpr int kBuckets = (27 + G - 1) / G;  // buckets whose ranges one lane reads
    static constexpr int kUnroll = 4;                  // candidate loads a lane has in flight
    static constexpr int kRuns = 64;                   // runs of up to 8 candidates listed at a time (a fluid at rest: ~40)
    static constexpr int kHits = 32 + kUnroll * G;     // hits listed before they are summed (a fluid at rest: ~27)
    static constexpr int kRow = G + 4;                 // one term of the G hits of a chunk; rows start in different banks
};

// NT rows of the terms of a chunk of G hits and a row of ones.
template <int G, int NT>
constexpr int kCoopTerms = (NT + 1) * CoopShape<G>::kRow;

// What a walk needs beside them.  Groups start G banks apart.
template <int G, int NT>
struct CoopMem {
    using S = CoopShape<G>;
    static constexpr int kPad = ((G - kCoopTerms<G, NT> - S::kHits - 2 * S::kRuns) % 32 + 32) % 32;
    float term[kCoopTerms<G, NT>];
    int2 run[S::kRuns];  // first candidate and candidates from there on in its bucket (a run takes up to 8)
    int hit[S::kHits + kPad];
};

// Terms alone, for the passes over kept hits.
template <int G, int NT>
struct CoopTermMem {
    static constexpr int kPad = ((G - kCoopTerms<G, NT>) % 32 + 32) % 32;
    float term[kCoopTerms<G, NT> + kPad];
};

// Hits of a particle in visiting order, kept from the lambda pass for the
// delta-p pass of the same iteration (the same positions, so the same hits).
constexpr uint32_t kNoHits = 0xFFFFFFFFu;

// The particle's sums: lane gl of a group adds t[ra] * t[rb] (fused) over the
// hits in order, row NT holding ones; load(k) reads hit k and pair(load(k), t)
// fills its terms (none for k = self).  The loads of U chunks of G hits are
// issued together.  Called by whole warps.
template <int G, int NT, int U, class Load, class Pair>
struct CoopSum {
    static constexpr int kRow = CoopShape<G>::kRow;
    float* term;
    int gl, self, ra, rb;
    float acc;
    Load load;
    Pair pair;
    __device__ __forceinline__ CoopSum(float* m, int lane_of_group, int s, int a, int b, float init, Load&& l, Pair&& p)
        : term(m), gl(lane_of_group), self(s), ra(a * kRow), rb(b * kRow), acc(init), load(l), pair(p)
    {
        term[NT * kRow + gl] = 1.0f;
    }
    // lane gl's hit k of a chunk (self: none); cnt hits in the chunk
    template <class D>
    __device__ __forceinline__ void chunk(int k, const D& d, int cnt)
    {
        float t[NT];
#pragma unroll
        for (int r = 0; r < NT; ++r) t[r] = 0.0f;
        if (k != self) pair(d, t);
#pragma unroll
        for (int r = 0; r < NT; ++r) term[r * kRow + gl] = t[r];
        __syncwarp();
#pragma unroll
        for (int q = 0; q < G; q += 4) {
            if (G > 8 && q >= cnt) break;
            const float4 a = *reinterpret_cast<const float4*>(term + ra + q);
            const float4 b = *reinterpret_cast<const float4*>(term + rb + q);
            acc = __fmaf_rn(a.x, b.x, acc);
            acc = __fmaf_rn(a.y, b.y, acc);
            acc = __fmaf_rn(a.z, b.z, acc);
            acc = __fmaf_rn(a.w, b.w, acc);
        }
        __syncwarp();
    }
    // cnt hits (per group), hit(i) = the i-th
    template <class HitAt>
    __device__ __forceinline__ void add(int cnt, HitAt&& hit)
    {
        const int most = (int)__reduce_max_sync(0xffffffffu, (uint32_t)cnt);
#pragma unroll 1
        for (int h = 0; h < most; h += U * G) {
            int k[U];
#pragma unroll
            for (int u = 0; u < U; ++u) k[u] = h + u * G + gl < cnt ? hit(h + u * G + gl) : self;
            decltype(load(0)) d[U];
#pragma unroll
            for (int u = 0; u < U; ++u) d[u] = load(k[u]);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (u > 0 && h + u * G >= most) break;
                chunk(k[u], d[u], cnt - h - u * G);
            }
        }
    }
    __device__ __forceinline__ float get(int k) const { return __shfl_sync(0xffffffffu, acc, k, G); }
};

// The walk of a particle whose hits were not kept, in a pass that otherwise
// reads kept hits: each[k] for its buckets' candidates G at a time, in
// visiting order (k = self where there is none).  Called by whole warps.
template <int G, class Each>
__device__ __forceinline__ void coop_plain_walk(const DevParams& P, const int2* __restrict__ table, uint32_t mask,
                                                const float4* __restrict__ X, float4 xi, int self, bool on, Each&& each)
{
    const int gl = threadIdx.x & (G - 1);
    const int cx = cell_coord(xi.x, P.h), cy = cell_coord(xi.y, P.h), cz = cell_coord(xi.z, P.h);
#pragma unroll 1
    for (int b = 0; b < 27; ++b) {
        int2 se = make_int2(0, 0);
        if (on) se = __ldg(table + grid_hash(cx + b % 3 - 1, cy + b / 3 % 3 - 1, cz + b / 9 - 1, mask));
        const int len = se.x == -1 ? 0 : se.y - se.x;
        const int most = (int)__reduce_max_sync(0xffffffffu, (uint32_t)len);
#pragma unroll 1
        for (int c = 0; c < most; c += G) {
            int k = self;
            if (c + gl < len) {
                const float4 xj = __ldg(X + se.x + c + gl);
                const float2 rxy = sub_f32x2(make_float2(xi.x, xi.y), make_float2(xj.x, xj.y));
                const float rx = rxy.x, ry = rxy.y, rz = xi.z - xj.z;
                if (rx * rx + ry * ry + rz * rz <= P.h2) k = se.x + c + gl;
            }
            each(k);
        }
    }
}

// One position per hit, and a second array's entry beside it.
struct CoopLoad1 {
    const float4* __restrict__ x;
    __device__ __forceinline__ float4 operator()(int k) const { return __ldg(x + k); }
};
struct CoopTwo {
    float4 x, v;
};
struct CoopLoad2 {
    const float4* __restrict__ x;
    const float4* __restrict__ v;
    __device__ __forceinline__ CoopTwo operator()(int k) const { return CoopTwo{__ldg(x + k), __ldg(v + k)}; }
};

// The candidates of 32 / G rounds as one word: bit r * G + l of the group's
// word is lane l's hit in round r.
template <int G>
__device__ __forceinline__ uint32_t coop_word(const uint32_t* bal, int lane)
{
    if constexpr (G == 32) {
        return bal[0];
    } else if constexpr (G == 16) {
        return __byte_perm(bal[0], bal[1], lane < 16 ? 0x5410 : 0x7632);
    } else {
        const uint32_t g = (uint32_t)lane >> 3, sel = g | (g + 4) << 4;
        return __byte_perm(__byte_perm(bal[0], bal[1], sel), __byte_perm(bal[2], bal[3], sel), 0x5410);
    }
}

// Walks the 27 buckets of the particle at xi: its hits, in visiting order and
// with the particle itself among them, go through sum.  Called by whole
// warps; a group without a particle passes live = false.  With `list` the hits
// are kept there (list_len = their number, or kNoHits where they do not fit).
template <int G, int NT, class Sum, class Hit>
__device__ __forceinline__ void coop_walk(const DevParams& P, const int2* __restrict__ table, uint32_t mask,
                                          const float4* __restrict__ X, float4 xi, bool live, CoopMem<G, NT>& M,
                                          Sum& sum, Hit&& hit, uint32_t* __restrict__ list, uint32_t* list_len)
{
    using S = CoopShape<G>;
    constexpr int kWord = 32 / G, kWords = S::kUnroll / kWord;  // rounds per word, words per step
    const int lane = threadIdx.x & 31, gl = lane & (G - 1);
    // bucket ranges: lane gl takes buckets gl, gl + G, ... of the visiting order
    // (the lanes' candidates then lie close in the list: fewer bank conflicts)
    int start[S::kBuckets], len[S::kBuckets], off[S::kBuckets], all = 0;
    const int cx = cell_coord(xi.x, P.h), cy = cell_coord(xi.y, P.h), cz = cell_coord(xi.z, P.h);
#pragma unroll
    for (int u = 0; u < S::kBuckets; ++u) {
        const int b = gl + u * G;
        int2 se = make_int2(0, 0);
        if (live && b < 27) {
            se = __ldg(table + grid_hash(cx + b % 3 - 1, cy + b / 3 % 3 - 1, cz + b / 9 - 1, mask));
            if (se.x == -1) se = make_int2(0, 0);
        }
        start[u] = se.x;
        len[u] = se.y - se.x;
    }
#pragma unroll
    for (int u = 0; u < S::kBuckets; ++u) {
        const int runs = (len[u] + 7) >> 3;
        int sum_to = runs;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, sum_to, o, G);
            if (gl >= o) sum_to += v;
        }
        off[u] = all + sum_to - runs;
        all += __shfl_sync(0xffffffffu, sum_to, G - 1, G);
    }

    const int all_max = (int)__reduce_max_sync(0xffffffffu, (uint32_t)all);
    int hits = 0, kept = 0;
    // the listed hits to the kept list and the sums
    auto flush = [&]() {
        __syncwarp();
        if (list)
            for (int i = gl; i < hits && kept + i < kCoopList; i += G) list[kept + i] = (uint32_t)M.hit[i];
        kept += hits;
        sum.add(hits, [&](int i) { return M.hit[i]; });
        hits = 0;
    };
    const int oct = gl >> 3, in_oct = lane & 7;
#pragma unroll 1
    for (int w0 = 0; w0 < all_max; w0 += S::kRuns) {
        // runs w0 .. w0 + kRuns - 1 of the 27 buckets, then empty ones
        __syncwarp();
        for (int r = 2 * gl; r < S::kRuns; r += 2 * G) *reinterpret_cast<int4*>(M.run + r) = make_int4(0, 0, 0, 0);
        __syncwarp();
#pragma unroll
        for (int u = 0; u < S::kBuckets; ++u) {
            int at = off[u] - w0;
            for (int c = 0; c < len[u]; c += 8, ++at)
                if ((uint32_t)at < (uint32_t)S::kRuns)
                    M.run[at] = make_int2(start[u] + c, len[u] - c);
        }
        __syncwarp();
        const int here_max = min(all_max - w0, S::kRuns);
#pragma unroll 1
        for (int base = 0; base < here_max; base += S::kUnroll * (G / 8)) {
            int k[S::kUnroll];
            float4 xj[S::kUnroll];
            uint32_t bal[S::kUnroll];
            bool h[S::kUnroll];
#pragma unroll
            for (int u = 0; u < S::kUnroll; ++u) {
                const int2 run = M.run[base + u * (G / 8) + oct];
                h[u] = in_oct < run.y;
                k[u] = run.x + in_oct;  // (kCoopPad slots past the arrays' end)
                xj[u] = __ldg(X + k[u]);
            }
#pragma unroll
            for (int u = 0; u < S::kUnroll; ++u) {
                const float2 rxy = sub_f32x2(make_float2(xi.x, xi.y), make_float2(xj[u].x, xj[u].y));
                const float rx = rxy.x, ry = rxy.y, rz = xi.z - xj[u].z;
                const float r2 = rx * rx + ry * ry + rz * rz;
                h[u] = h[u] && hit(r2);
                bal[u] = __ballot_sync(0xffffffffu, h[u]);
            }
#pragma unroll
            for (int w = 0; w < kWords; ++w) {
                const uint32_t word = coop_word<G>(bal + w * kWord, lane);
#pragma unroll
                for (int u = 0; u < kWord; ++u) {
                    const uint32_t below = ((1u << gl) - 1u) << (u * G) | ((1u << (u * G)) - 1u);
                    if (h[w * kWord + u]) M.hit[hits + __popc(word & below)] = k[w * kWord + u];
                }
                hits += __popc(word);
            }
            if (__any_sync(0xffffffffu, hits > 32)) flush();
        }
    }
    flush();
    if (list) *list_len = kept <= kCoopList ? (uint32_t)kept : kNoHits;
}

// The particle of a group: its processing index t (scene lookup), slot s.
struct CoopParticle {
    bool live;
    int t, s;
};
template <int G>
__device__ __forceinline__ CoopParticle coop_particle(uint32_t n, const uint32_t* __restrict__ order)
{
    const uint32_t t = (blockIdx.x * kCThreads + threadIdx.x) / G;
    CoopParticle c;
    c.live = t < n;
    c.t = c.live ? (int)t : 0;
    c.s = order ? (int)__ldg(order + c.t) : c.t;
    return c;
}

// row index of lane gl's sum: nibble gl of `rows`
__device__ __forceinline__ int coop_row(uint32_t rows, int gl) { return gl < 8 ? (int)(rows >> (4 * gl) & 15u) : 0; }

}  // namespace pbf
