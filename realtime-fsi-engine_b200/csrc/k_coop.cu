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
#include <type_traits>

#include "coop_walk.cuh"
#include "pbf_batch.h"

namespace pbf {

template <int G, bool B>
__global__ void __launch_bounds__(kCThreads, kCBlocks) k_c_lambda(DevParams P, const SceneDev* __restrict__ scenes,
                                                        const uint16_t* __restrict__ scene_of,
                                                        const float4* __restrict__ xin, float4* __restrict__ xout,
                                                        float* __restrict__ rho_out, const int2* __restrict__ table,
                                                        const uint32_t* __restrict__ lod, uint32_t iter,
                                                        const uint32_t* __restrict__ order,
                                                        uint32_t* __restrict__ list, uint32_t* __restrict__ list_len,
                                                        float4* __restrict__ aux)
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
    auto pair = [&](float4 xj, float(&t)[NT]) {
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
    CoopSum<G, NT, 1, CoopLoad1, decltype(pair)> sum(M.term, gl, s, coop_row(0x43243210u, gl), coop_row(0x55566666u, gl),
                                                  gl == 0 ? P.w0_self : 0.0f, CoopLoad1{xin}, std::move(pair));
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
    if (aux) aux[s] = make_float4(gc.x, gc.y, gc.z, den);
}

// W: no hits are kept for any particle
template <int G, bool B, bool W = false>
__global__ void __launch_bounds__(kCThreads, kReplayBlocks) k_c_deltap(DevParams P, const SceneDev* __restrict__ scenes,
                                                        const uint16_t* __restrict__ scene_of,
                                                        const float4* __restrict__ xin, float4* __restrict__ xout,
                                                        const int2* __restrict__ table,
                                                        const uint32_t* __restrict__ lod, uint32_t iter,
                                                        const uint32_t* __restrict__ order,
                                                        const uint32_t* __restrict__ list,
                                                        const uint32_t* __restrict__ list_len,
                                                        float4* __restrict__ dp_out)
{
    constexpr int NT = 4;
    __shared__ __align__(16) std::conditional_t<W, CoopMem<G, NT>, CoopTermMem<G, NT>> mem[kCThreads / G];
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
    auto pair = [&](float4 xj, float(&t)[NT]) {
        const float2 rxy = sub_f32x2(make_float2(xi.x, xi.y), make_float2(xj.x, xj.y));
        const float rx = rxy.x, ry = rxy.y, rz = xi.z - xj.z;
        const float r2 = rx * rx + ry * ry + rz * rz;
        if (!(r2 >= 1e-10f)) return;
        t[0] = rx;
        t[1] = ry;
        t[2] = rz;
        t[3] = spiky_scale(P, r2) * xj.w;
    };
    // sums: lambda_j gradW xyz, from the lambda pass's part on
    CoopSum<G, NT, W ? 1 : kReplayAhead, CoopLoad1, decltype(pair)> sum(
        mem[threadIdx.x / G].term, gl, s, min(gl, 2), 3, gl == 0 ? b.x : gl == 1 ? b.y : b.z, CoopLoad1{xin},
        std::move(pair));
    const bool on = c.live && !skip;
    if constexpr (W) {
        coop_walk<G, NT>(P, table, mask, xin, xi, on, mem[threadIdx.x / G], sum, [&](float r2) { return r2 <= P.h2; },
                         nullptr, nullptr);
    } else {
        const uint32_t len = on && list ? __ldg(list_len + s) : kNoHits;
        if (__any_sync(0xffffffffu, on && len == kNoHits))
            coop_plain_walk<G>(P, table, mask, xin, xi, s, on && len == kNoHits,
                               [&](int k) { sum.chunk(k, __ldg(xin + k), G); });
        const uint32_t* mine = list + (size_t)s * kCoopList;
        sum.add(len == kNoHits ? 0 : (int)len, [&](int i) { return (int)__ldg(mine + i); });
    }
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
    if (dp_out) dp_out[s] = make_float4(dp.x, dp.y, dp.z, 0.f);
}

template <int G, bool B>
__global__ void __launch_bounds__(kCThreads, kCBlocks) k_c_integrate(DevParams P, const SceneDev* __restrict__ scenes,
                                                           const uint16_t* __restrict__ scene_of,
                                                           const float4* __restrict__ xs,
                                                           const float4* __restrict__ sv, float4* __restrict__ sx0,
                                                           float4* __restrict__ somega,
                                                           const uint32_t* __restrict__ ids, float4* __restrict__ pos,
                                                           float4* __restrict__ vel, const int2* __restrict__ table,
                                                           const uint32_t* __restrict__ order,
                                                           uint32_t* __restrict__ list,
                                                           uint32_t* __restrict__ list_len,
                                                           float4* __restrict__ fsum)
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
    auto pair = [&](CoopTwo j, float(&t)[NT]) {
        const float4 xj = j.x, vj = j.v;
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
    CoopSum<G, NT, 1, CoopLoad2, decltype(pair)> sum(M.term, gl, s, coop_row(0x00654210u, gl), coop_row(0x77777333u, gl), 0.0f,
                                                  CoopLoad2{xs, sv}, std::move(pair));
    uint32_t len = kNoHits;
    coop_walk<G, NT>(P, table, mask, xs, x4, c.live && (P.visc_on || P.vort_on), M, sum,
                     [&](float r2) { return r2 <= P.h2; }, c.live && list ? list + (size_t)s * kCoopList : nullptr,
                     &len);
    const float3 f = make_float3(sum.get(0), sum.get(1), sum.get(2));
    const float3 cu = make_float3(sum.get(3), sum.get(4), sum.get(5));
    if (!c.live || gl != 0) return;
    if (list) list_len[s] = len;
    if (fsum) fsum[s] = make_float4(f.x, f.y, f.z, 0.f);
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
    auto pair = [&](CoopTwo j, float(&t)[NT]) {
        const float4 xj = j.x;
        const float2 rxy = sub_f32x2(make_float2(xi.x, xi.y), make_float2(xj.x, xj.y));
        const float rx = rxy.x, ry = rxy.y, rz = xi.z - xj.z;
        const float r2 = rx * rx + ry * ry + rz * rz;
        t[0] = rx;
        t[1] = ry;
        t[2] = rz;
        t[3] = spiky_scale(P, r2) * j.v.w;
    };
    // sums: |omega_j| gradW xyz
    CoopMem<G, NT>& M = mem[threadIdx.x / G];
    CoopSum<G, NT, 1, CoopLoad2, decltype(pair)> sum(M.term, gl, s, min(gl, 2), 3, 0.0f, CoopLoad2{spos, somega},
                                                  std::move(pair));
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

// Passes over kept hits need no walk, and three or four sums: four lanes keep
// more of the warp at work (131,072 particles: delta-p 22.5 us against 27.8
// with 8 lanes, the reverse delta-p 31.6 against 34.4; 32,768: 8.2 against 10.0,
// 12.6 against 12.9).
int coop_replay_lanes(int G, uint32_t n) { return n > 16384u ? 4 : G; }

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
                     const uint32_t* order, uint32_t* list, uint32_t* list_len, float4* aux, cudaStream_t st)
{
    PBF_COOP_LAUNCH(k_c_lambda, P, scenes, scene_of, xin, xout, rho, table, lod, iter, order, list, list_len, aux);
}

void launch_c_deltap(int G, const DevParams& P, const SceneDev* scenes, const uint16_t* scene_of, const float4* xin,
                     float4* xout, const int2* table, const uint32_t* lod, uint32_t iter, const uint32_t* order,
                     const uint32_t* list, const uint32_t* list_len, float4* dp_out, cudaStream_t st)
{
    G = coop_replay_lanes(G, P.n);
    if (scenes && !list) {  // an adjoint's record without hits
        k_c_deltap<8, true, true><<<cgrid(P.n, 8), kCThreads, 0, st>>>(P, scenes, scene_of, xin, xout, table, lod, iter,
                                                                       order, list, list_len, dp_out);
        return;
    }
    if (G == 4) {
        if (scenes)
            k_c_deltap<4, true><<<cgrid(P.n, 4), kCThreads, 0, st>>>(P, scenes, scene_of, xin, xout, table, lod, iter,
                                                                     order, list, list_len, dp_out);
        else
            k_c_deltap<4, false><<<cgrid(P.n, 4), kCThreads, 0, st>>>(P, scenes, scene_of, xin, xout, table, lod, iter,
                                                                      order, list, list_len, dp_out);
        return;
    }
    PBF_COOP_LAUNCH(k_c_deltap, P, scenes, scene_of, xin, xout, table, lod, iter, order, list, list_len, dp_out);
}

void launch_c_integrate(int G, const DevParams& P, const SceneDev* scenes, const uint16_t* scene_of, const float4* xs,
                        const float4* sv, float4* sx0, float4* somega, const uint32_t* ids, float4* pos, float4* vel,
                        const int2* table, const uint32_t* order, uint32_t* list, uint32_t* list_len, float4* fsum,
                        cudaStream_t st)
{
    PBF_COOP_LAUNCH(k_c_integrate, P, scenes, scene_of, xs, sv, sx0, somega, ids, pos, vel, table, order, list, list_len,
                    fsum);
}

void launch_c_vorticity(int G, const DevParams& P, const SceneDev* scenes, const uint16_t* scene_of,
                        const float4* spos, const float4* somega, const uint32_t* ids, float4* vel, const int2* table,
                        const uint32_t* order, cudaStream_t st)
{
    PBF_COOP_LAUNCH(k_c_vorticity, P, scenes, scene_of, spos, somega, ids, vel, table, order);
}

#undef PBF_COOP_LAUNCH

}  // namespace pbf
