// k_coop.cu — neighbour passes over the hashed buckets with a group of G
// lanes per particle, for scenes too small to fill the GPU with one thread
// per particle.
//
// One thread walking 27 buckets is a chain of some hundred dependent loads
// and pair bodies; a small scene has a few warps per SM and waits for that
// chain (52 us for a lambda pass of 2,197 particles, 72 us at 32,768).  Here
// the lanes of a group read the buckets' ranges together, lay the candidates
// out in one list in the reference's visiting order, test G at a time into a
// compacted list of hits, and evaluate one hit per lane.  The sums stay the
// sequential ones: the lanes' pair terms go through shared memory and one
// lane per sum adds them in visiting order with the roundings of the
// one-thread bodies (masked_body.cuh), so every result has their bits.
#include "masked_body.cuh"
#include "pbf_batch.h"
#include "pbf_kernels.h"
#include <utility>

namespace pbf {

constexpr int kCThreads = 128;
// 8 resident blocks (64 registers): the lists of a block take 13-16 KB of the
// SM's 256 KB of shared memory and L1, and what is left over caches the
// neighbours' positions, so more residency does not pay (a lambda pass of
// 32,768 particles at G = 8: 22.4 us; 6 blocks: 23.0, 10: 24.7, 12: 29.3).
constexpr int kCBlocks = 8;

template <int G>
struct CoopShape {
    static constexpr int kBuckets = (27 + G - 1) / G;  // buckets whose ranges one lane reads
    static constexpr int kUnroll = 4;                  // candidate loads a lane has in flight
    static constexpr int kRuns = 64;                   // runs of up to 8 candidates listed at a time (a fluid at rest: ~40)
    static constexpr int kHits = 32 + kUnroll * G;     // hits listed before they are summed (a fluid at rest: ~27)
    static constexpr int kRow = G + 4;                 // one term of the G hits of a chunk; rows start in different banks
};

// NT rows of pair terms and a row of ones.  Groups start G banks apart.
template <int G, int NT>
struct CoopMem {
    using S = CoopShape<G>;
    static constexpr int kTerms = (NT + 1) * S::kRow;
    static constexpr int kPad = ((G - kTerms - S::kHits - 2 * S::kRuns) % 32 + 32) % 32;
    float term[kTerms];
    int2 run[S::kRuns];  // first candidate and candidates from there on in its bucket (a run takes up to 8)
    int hit[S::kHits + kPad];
};

// Hits of a particle in visiting order, kept from the lambda pass for the
// delta-p pass of the same iteration (the same positions, so the same hits).
constexpr uint32_t kNoHits = 0xFFFFFFFFu;

// The particle's sums: lane gl of a group adds t[ra] * t[rb] (fused) over the
// hits in order, row NT holding ones; pair(k, t) fills the terms of hit k.
// Called by whole warps.
template <int G, int NT, class Pair>
struct CoopSum {
    using S = CoopShape<G>;
    CoopMem<G, NT>& M;
    int gl, ra, rb;
    float acc;
    Pair pair;
    __device__ __forceinline__ CoopSum(CoopMem<G, NT>& m, int lane_of_group, int a, int b, float init, Pair&& p)
        : M(m), gl(lane_of_group), ra(a * S::kRow), rb(b * S::kRow), acc(init), pair(p)
    {
        M.term[NT * S::kRow + gl] = 1.0f;
    }
    // cnt hits (per group), hit(i) = the i-th
    template <class HitAt>
    __device__ __forceinline__ void add(int cnt, HitAt&& hit)
    {
        const int most = (int)__reduce_max_sync(0xffffffffu, (uint32_t)cnt);
#pragma unroll 1
        for (int h = 0; h < most; h += G) {
            float t[NT];
#pragma unroll
            for (int r = 0; r < NT; ++r) t[r] = 0.0f;
            if (h + gl < cnt) pair(hit(h + gl), t);
#pragma unroll
            for (int r = 0; r < NT; ++r) M.term[r * S::kRow + gl] = t[r];
            __syncwarp();
#pragma unroll
            for (int q = 0; q < G; q += 4) {
                if (G > 8 && h + q >= cnt) break;
                const float4 a = *reinterpret_cast<const float4*>(M.term + ra + q);
                const float4 b = *reinterpret_cast<const float4*>(M.term + rb + q);
                acc = __fmaf_rn(a.x, b.x, acc);
                acc = __fmaf_rn(a.y, b.y, acc);
                acc = __fmaf_rn(a.z, b.z, acc);
                acc = __fmaf_rn(a.w, b.w, acc);
            }
            __syncwarp();
        }
    }
    __device__ __forceinline__ float get(int k) const { return __shfl_sync(0xffffffffu, acc, k, G); }
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

template <int G, bool B>
__global__ void __launch_bounds__(kCThreads, kCBlocks) k_c_lambda(DevParams P, const SceneDev* __restrict__ scenes,
                                                        const uint16_t* __restrict__ scene_of,
                                                        const float4* __restrict__ xin, float4* __restrict__ xout,
                                                        float* __restrict__ rho_out, const int2* __restrict__ table,
                                                        const uint32_t* __restrict__ lod, uint32_t iter,
                                                        const uint32_t* __restrict__ order,
                                                        uint32_t* __restrict__ list, uint32_t* __restrict__ list_len)
{
    constexpr int NT = 6;
    __shared__ __align__(16) CoopMem<G, NT> mem[kCThreads / G];
    const CoopParticle c = coop_particle<G>(P.n, order);
    const int gl = threadIdx.x & (G - 1), s = c.s;
    const float4 xi = __ldg(xin + s);
    const bool skip = P.apbf && __ldg(lod + s) < iter;
    uint32_t mask = P.mask;
    if constexpr (B) {
        const SceneDev* S = scenes + __ldg(scene_of + c.t);
        table += __ldg(&S->table_off);
        mask = __ldg(&S->mask);
    }
    const bool scorr = P.scorr && P.wq > 1e-12f;
    auto pair = [&](int k, float(&t)[NT]) {
        if (k == s) return;
        const float4 xj = __ldg(xin + k);
        const float2 rxy = sub_f32x2(make_float2(xi.x, xi.y), make_float2(xj.x, xj.y));
        const float rx = rxy.x, ry = rxy.y, rz = xi.z - xj.z;
        const float r2 = rx * rx + ry * ry + rz * rz;
        const float w = poly6_in(P, r2);
        t[0] = w;
        if (r2 >= 1e-10f) {
            const float sc = spiky_scale(P, r2);
            const float2 axy = mul_f32x2(rxy, sc);
            const float ax = axy.x, ay = axy.y, az = rz * sc;
            t[1] = ax * ax + ay * ay + az * az;
            t[2] = ax;
            t[3] = ay;
            t[4] = az;
            if (scorr) {
                const float ratio = w * P.inv_wq;
                float pw;
                if (P.ncorr_is4) {
                    const float q = ratio * ratio;
                    pw = q * q;
                } else {
                    pw = powf(ratio, P.n_corr);
                }
                t[5] = pw;
            }
        }
    };
    // sums: rho, |gradW|^2, gradW xyz, (W / W(dq))^n gradW xyz
    CoopMem<G, NT>& M = mem[threadIdx.x / G];
    CoopSum<G, NT, decltype(pair)> sum(M, gl, coop_row(0x43243210u, gl), coop_row(0x55566666u, gl),
                                       gl == 0 ? P.w0_self : 0.0f, std::move(pair));
    uint32_t len = kNoHits;
    coop_walk<G, NT>(P, table, mask, xin, xi, c.live && !skip, M, sum, [&](float r2) { return r2 <= P.h2; },
                     c.live && list ? list + (size_t)s * kCoopList : nullptr, &len);
    const float rho = sum.get(0), sg = sum.get(1);
    const float3 g = make_float3(sum.get(2), sum.get(3), sum.get(4));
    const float3 sc = make_float3(sum.get(5), sum.get(6), sum.get(7));
    if (!c.live || gl != 0) return;
    if (list) list_len[s] = len;
    if (skip) {
        xout[s] = xi;
        return;
    }
    float rho_, den;
    float3 gc, b;
    xout[s] = lambda_finish(P, xi, rho, sg, g, sc, scorr, rho_, gc, den, b);
    rho_out[s] = rho_;
    P.dpb[s] = make_float4(b.x, b.y, b.z, 0.f);
}

template <int G, bool B>
__global__ void __launch_bounds__(kCThreads, kCBlocks) k_c_deltap(DevParams P, const SceneDev* __restrict__ scenes,
                                                        const uint16_t* __restrict__ scene_of,
                                                        const float4* __restrict__ xin, float4* __restrict__ xout,
                                                        const int2* __restrict__ table,
                                                        const uint32_t* __restrict__ lod, uint32_t iter,
                                                        const uint32_t* __restrict__ order,
                                                        const uint32_t* __restrict__ list,
                                                        const uint32_t* __restrict__ list_len)
{
    constexpr int NT = 4;
    __shared__ __align__(16) CoopMem<G, NT> mem[kCThreads / G];
    const CoopParticle c = coop_particle<G>(P.n, order);
    const int gl = threadIdx.x & (G - 1), s = c.s;
    const float4 xi = __ldg(xin + s);
    const bool skip = P.apbf && __ldg(lod + s) < iter;
    uint32_t mask = P.mask;
    const SceneDev* S = nullptr;
    if constexpr (B) {
        S = scenes + __ldg(scene_of + c.t);
        table += __ldg(&S->table_off);
        mask = __ldg(&S->mask);
    }
    const float4 b = __ldg(P.dpb + s);
    auto pair = [&](int k, float(&t)[NT]) {
        const float4 xj = __ldg(xin + k);
        const float2 rxy = sub_f32x2(make_float2(xi.x, xi.y), make_float2(xj.x, xj.y));
        const float rx = rxy.x, ry = rxy.y, rz = xi.z - xj.z;
        const float r2 = rx * rx + ry * ry + rz * rz;
        if (k == s || !(r2 >= 1e-10f)) return;
        t[0] = rx;
        t[1] = ry;
        t[2] = rz;
        t[3] = spiky_scale(P, r2) * xj.w;
    };
    // sums: lambda_j gradW xyz, from the lambda pass's part on
    CoopMem<G, NT>& M = mem[threadIdx.x / G];
    CoopSum<G, NT, decltype(pair)> sum(M, gl, min(gl, 2), 3, gl == 0 ? b.x : gl == 1 ? b.y : b.z, std::move(pair));
    const bool on = c.live && !skip;
    const uint32_t len = on && list ? __ldg(list_len + s) : kNoHits;
    if (__any_sync(0xffffffffu, on && len == kNoHits))
        coop_walk<G, NT>(P, table, mask, xin, xi, on && len == kNoHits, M, sum,
                         [&](float r2) { return r2 <= P.h2 && r2 >= 1e-10f; }, nullptr, nullptr);
    const uint32_t* mine = list + (size_t)s * kCoopList;
    sum.add(len == kNoHits ? 0 : (int)len, [&](int i) { return (int)__ldg(mine + i); });
    const float3 d = make_float3(sum.get(0), sum.get(1), sum.get(2));
    if (!c.live || gl != 0) return;
    if (skip) {
        xout[s] = xi;
        return;
    }
    float3 dp;
    if constexpr (B)
        xout[s] = deltap_finish(P, load_sdf(S), xi, d, dp);
    else
        xout[s] = deltap_finish(P, P.sdf, xi, d, dp);
}

template <int G, bool B>
__global__ void __launch_bounds__(kCThreads, kCBlocks) k_c_integrate(DevParams P, const SceneDev* __restrict__ scenes,
                                                           const uint16_t* __restrict__ scene_of,
                                                           const float4* __restrict__ xs,
                                                           const float4* __restrict__ sv, float4* __restrict__ sx0,
                                                           float4* __restrict__ somega,
                                                           const uint32_t* __restrict__ ids, float4* __restrict__ pos,
                                                           float4* __restrict__ vel, const int2* __restrict__ table,
                                                           const uint32_t* __restrict__ order)
{
    constexpr int NT = 7;
    __shared__ __align__(16) CoopMem<G, NT> mem[kCThreads / G];
    const CoopParticle c = coop_particle<G>(P.n, order);
    const int gl = threadIdx.x & (G - 1), s = c.s;
    const float4 x4 = __ldg(xs + s);
    const float4 v0 = __ldg(sv + s);
    uint32_t mask = P.mask;
    const SceneDev* S = nullptr;
    if constexpr (B) {
        S = scenes + __ldg(scene_of + c.t);
        table += __ldg(&S->table_off);
        mask = __ldg(&S->mask);
    }
    auto pair = [&](int k, float(&t)[NT]) {
        if (k == s) return;
        const float4 xj = __ldg(xs + k);
        const float4 vj = __ldg(sv + k);
        const float2 rxy = sub_f32x2(make_float2(x4.x, x4.y), make_float2(xj.x, xj.y));
        const float rx = rxy.x, ry = rxy.y, rz = x4.z - xj.z;
        const float r2 = rx * rx + ry * ry + rz * rz;
        const float2 uxy = sub_f32x2(make_float2(vj.x, vj.y), make_float2(v0.x, v0.y));
        const float ux = uxy.x, uy = uxy.y, uz = vj.z - v0.z;
        t[0] = ux;
        t[1] = uy;
        t[2] = uz;
        if (P.visc_on) t[3] = poly6_in(P, r2) * P.inv_rho0;
        if (P.vort_on && r2 >= 1e-10f) {
            const float sc = spiky_scale(P, r2);
            const float2 axy = mul_f32x2(rxy, sc);
            const float ax = axy.x, ay = axy.y, az = rz * sc;
            t[4] = __fmaf_rn(uy, az, -__fmul_rn(uz, ay));
            t[5] = __fmaf_rn(uz, ax, -__fmul_rn(ux, az));
            t[6] = __fmaf_rn(ux, ay, -__fmul_rn(uy, ax));
        }
    };
    // sums: W u xyz, u x gradW xyz
    CoopMem<G, NT>& M = mem[threadIdx.x / G];
    CoopSum<G, NT, decltype(pair)> sum(M, gl, coop_row(0x00654210u, gl), coop_row(0x77777333u, gl), 0.0f,
                                       std::move(pair));
    coop_walk<G, NT>(P, table, mask, xs, x4, c.live && (P.visc_on || P.vort_on), M, sum,
                     [&](float r2) { return r2 <= P.h2; }, nullptr, nullptr);
    const float3 f = make_float3(sum.get(0), sum.get(1), sum.get(2));
    const float3 cu = make_float3(sum.get(3), sum.get(4), sum.get(5));
    if (!c.live || gl != 0) return;
    float4 xo, vo, om;
    if constexpr (B) {
        float bmin[3], bmax[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            bmin[a] = __ldg(&S->bmin[a]);
            bmax[a] = __ldg(&S->bmax[a]);
        }
        integrate_finish(P, bmin, bmax, load_sdf(S), x4, v0, sx0[s], f, cu, xo, vo, om);
    } else {
        integrate_finish(P, P.bmin, P.bmax, P.sdf, x4, v0, sx0[s], f, cu, xo, vo, om);
    }
    if (P.vort_on) somega[s] = om;
    const uint32_t id = __ldg(ids + s);
    pos[id] = xo;
    vel[id] = vo;
    sx0[s] = xo;
}

template <int G, bool B>
__global__ void __launch_bounds__(kCThreads, kCBlocks) k_c_vorticity(DevParams P, const SceneDev* __restrict__ scenes,
                                                           const uint16_t* __restrict__ scene_of,
                                                           const float4* __restrict__ spos,
                                                           const float4* __restrict__ somega,
                                                           const uint32_t* __restrict__ ids, float4* __restrict__ vel,
                                                           const int2* __restrict__ table,
                                                           const uint32_t* __restrict__ order)
{
    constexpr int NT = 4;
    __shared__ __align__(16) CoopMem<G, NT> mem[kCThreads / G];
    const CoopParticle c = coop_particle<G>(P.n, order);
    const int gl = threadIdx.x & (G - 1), s = c.s;
    const float4 xi = __ldg(spos + s);
    uint32_t mask = P.mask;
    if constexpr (B) {
        const SceneDev* S = scenes + __ldg(scene_of + c.t);
        table += __ldg(&S->table_off);
        mask = __ldg(&S->mask);
    }
    auto pair = [&](int k, float(&t)[NT]) {
        if (k == s) return;
        const float4 xj = __ldg(spos + k);
        const float m = __ldg(&somega[k].w);
        const float2 rxy = sub_f32x2(make_float2(xi.x, xi.y), make_float2(xj.x, xj.y));
        const float rx = rxy.x, ry = rxy.y, rz = xi.z - xj.z;
        const float r2 = rx * rx + ry * ry + rz * rz;
        t[0] = rx;
        t[1] = ry;
        t[2] = rz;
        t[3] = spiky_scale(P, r2) * m;
    };
    // sums: |omega_j| gradW xyz
    CoopMem<G, NT>& M = mem[threadIdx.x / G];
    CoopSum<G, NT, decltype(pair)> sum(M, gl, min(gl, 2), 3, 0.0f, std::move(pair));
    coop_walk<G, NT>(P, table, mask, spos, xi, c.live, M, sum, [&](float r2) { return r2 <= P.h2 && r2 >= 1e-10f; },
                     nullptr, nullptr);
    const float3 e = make_float3(sum.get(0), sum.get(1), sum.get(2));
    if (!c.live || gl != 0) return;
    float3 dv;
    if (!vorticity_finish(P, e, [&] { return __ldg(somega + s); }, dv)) return;
    const uint32_t id = __ldg(ids + s);
    float4 v = vel[id];
    v.x += dv.x;
    v.y += dv.y;
    v.z += dv.z;
    vel[id] = v;
}

// ---- launchers -----------------------------------------------------------------------------
// One step (2 substeps of 4 iterations, a moving block, graph replay) with 32 /
// 16 / 8 lanes per particle and with one thread per particle, microseconds:
// 1,000 particles 157 / 173 / 195 / 835; 4,096 186 / 192 / 219 / 1005; 8,000
// 250 / 219 / 237 / 1122; 12,167 305 / 287 / 263 / 1167; 64,000 986 / 762 / 690
// / 1471; 180,000 2573 / 1914 / 1653 / 2301; 262,144 3699 / 2729 / 2335 / 3496.
// At 0.6M particles of an orderly fluid (one substep) 8 lanes take 2470 and one
// thread 2060: there the threads' shared loads win.
int coop_lanes(uint32_t n)
{
    if (n <= 4096u) return 32;
    if (n <= 8192u) return 16;
    return n <= (1u << 18) ? 8 : 0;
}

static inline unsigned cgrid(uint32_t n, int G)
{
    return (unsigned)(((uint64_t)n * (uint64_t)G + kCThreads - 1) / kCThreads);
}

#define PBF_COOP_LAUNCH(KERNEL, ...)                                                               \
    do {                                                                                          \
        if (scenes) {                                                                             \
            if (G == 32) KERNEL<32, true><<<cgrid(P.n, 32), kCThreads, 0, st>>>(__VA_ARGS__);     \
            else if (G == 16) KERNEL<16, true><<<cgrid(P.n, 16), kCThreads, 0, st>>>(__VA_ARGS__); \
            else KERNEL<8, true><<<cgrid(P.n, 8), kCThreads, 0, st>>>(__VA_ARGS__);               \
        } else {                                                                                  \
            if (G == 32) KERNEL<32, false><<<cgrid(P.n, 32), kCThreads, 0, st>>>(__VA_ARGS__);    \
            else if (G == 16) KERNEL<16, false><<<cgrid(P.n, 16), kCThreads, 0, st>>>(__VA_ARGS__); \
            else KERNEL<8, false><<<cgrid(P.n, 8), kCThreads, 0, st>>>(__VA_ARGS__);              \
        }                                                                                         \
    } while (0)

void launch_c_lambda(int G, const DevParams& P, const SceneDev* scenes, const uint16_t* scene_of, const float4* xin,
                     float4* xout, float* rho, const int2* table, const uint32_t* lod, uint32_t iter,
                     const uint32_t* order, uint32_t* list, uint32_t* list_len, cudaStream_t st)
{
    PBF_COOP_LAUNCH(k_c_lambda, P, scenes, scene_of, xin, xout, rho, table, lod, iter, order, list, list_len);
}

void launch_c_deltap(int G, const DevParams& P, const SceneDev* scenes, const uint16_t* scene_of, const float4* xin,
                     float4* xout, const int2* table, const uint32_t* lod, uint32_t iter, const uint32_t* order,
                     const uint32_t* list, const uint32_t* list_len, cudaStream_t st)
{
    PBF_COOP_LAUNCH(k_c_deltap, P, scenes, scene_of, xin, xout, table, lod, iter, order, list, list_len);
}

void launch_c_integrate(int G, const DevParams& P, const SceneDev* scenes, const uint16_t* scene_of, const float4* xs,
                        const float4* sv, float4* sx0, float4* somega, const uint32_t* ids, float4* pos, float4* vel,
                        const int2* table, const uint32_t* order, cudaStream_t st)
{
    PBF_COOP_LAUNCH(k_c_integrate, P, scenes, scene_of, xs, sv, sx0, somega, ids, pos, vel, table, order);
}

void launch_c_vorticity(int G, const DevParams& P, const SceneDev* scenes, const uint16_t* scene_of,
                        const float4* spos, const float4* somega, const uint32_t* ids, float4* vel, const int2* table,
                        const uint32_t* order, cudaStream_t st)
{
    PBF_COOP_LAUNCH(k_c_vorticity, P, scenes, scene_of, spos, somega, ids, vel, table, order);
}

#undef PBF_COOP_LAUNCH

}  // namespace pbf
