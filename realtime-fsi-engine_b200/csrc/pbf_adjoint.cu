// pbf_adjoint.cu — differentiable step of the multi-scene engine.
//
// pbf_batch_forward_record runs one step (every substep, then vorticity)
// exactly as pbf_batch_step does, saving the particle state at the start of
// each substep and, where memory allows, everything the reverse passes read of
// it: the sort permutation and cell table (replayed, not differentiated), (x*,
// lambda), the lambda denominators, the raw dp and the particles' hits of every
// iteration.  pbf_batch_backward walks the substeps
// in reverse with the kernels of k_adjoint.cu: vorticity (last substep),
// integrate, (deltaP+apply, lambda) per iteration, predict.  Without the room,
// or when a scene changed since the recording, it first runs each substep's
// forward again from its checkpoint, and with room for no hits either its
// passes walk the buckets again.  Gradients are with respect to the
// initial positions and velocities and each scene's SDF translation.  Both
// sequences are captured once into CUDA graphs.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <type_traits>

#include "../../include/pbf_b200.h"
#include "pbf_batch.h"
#include "pbf_engine.h"

using namespace pbf;

#define ACK(call)                                                                                  \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            return pbf::set_error(PBF_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(e_));   \
    } while (0)

template <class T>
static int aalloc(T*& p, size_t count)
{
    if (p) cudaFree(p);
    p = nullptr;
    if (count == 0) count = 1;
    cudaError_t e = cudaMalloc((void**)&p, count * sizeof(T));
    if (e != cudaSuccess) {
        p = nullptr;
        cudaGetLastError();  // (else the next launch's check reports it again)
        return set_error(PBF_ERR_ALLOC, "cudaMalloc(%zu B): %s", count * sizeof(T), cudaGetErrorString(e));
    }
    return PBF_OK;
}

template <class T>
static void afree(T*& p)
{
    if (p) cudaFree(p);
    p = nullptr;
}

void pbf_batch::ad_free()
{
    afree(ad_slab);
    ad_arrays.release();
    records.clear();
    ad_sx0 = ad_om = nullptr;
    ad_subs = ad_iters = 0;
    recorded = false;
}

// Lanes per particle of the recording and reverse passes: groups at any size
// (524,288 particles in 16 scenes, per iteration: recording 322 us and reverse
// 191, one thread per particle 278 and 361).
int pbf_batch::ad_lanes() const { return std::max(coop_lanes(n), 8); }

// One record's arrays laid one after another from `base` (null: only counted);
// returns its bytes.  `c` entries per array (a multiple of 64, pads included).
// Without hits (and so recomputed before each use) it holds what the
// iterations leave; the rest stays in the batch's own arrays of a substep (fsum
// in the lambda pass's part of delta-p, which an integrate pass does not read).
static size_t lay_record(pbf_batch& b, pbf_batch::Record& r, char* base, size_t c, uint32_t iters, bool hits)
{
    size_t at = 0;
    auto take = [&](auto*& p, size_t count) {
        p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(base + at);
        at += (count * sizeof(*p) + 255) / 256 * 256;
    };
    take(r.xl, c * iters);
    take(r.auxl, c * iters);
    take(r.auxd, c * iters);
    take(r.rhol, c * iters);
    if (hits) {
        take(r.ids, c);
        take(r.table, b.table_size);
        take(r.sv, c);
        take(r.xf, c);
        take(r.fsum, c);
        take(r.list, c * (iters + 1) * kCoopList);
        take(r.list_len, c * (iters + 1));
    } else {
        r.ids = b.ia;
        r.table = b.table;
        r.sv = b.sv;
        r.xf = b.sx[0];
        r.fsum = b.dpb;
        r.list = r.list_len = nullptr;
    }
    return at;
}

int pbf_batch::ad_alloc()
{
    const uint32_t S = cfg.substep_iterations, I = cfg.solver_iterations;
    if (ad_subs == S && ad_iters == I && cp_pos) return PBF_OK;
    ad_free();
    const size_t c = std::max<uint32_t>(n, 1u);
    int rc;
    ad_arrays.add(cp_pos, c * S).add(cp_vel, c * S).add(gxa, c).add(gxb, c).add(gv, c).add(x0b, c).add(pb, c).add(vb, c)
        .add(pbs, c).add(omb, c).add(tpos, c).add(tvel, c).add(tgrad, 4 * scenes.size());
    if ((rc = ad_arrays.alloc())) return rc;
    // A record per substep when they take at most a quarter of the free memory
    // (32,768 particles x 16 substeps x 4 iterations: 0.9 GB), else one when it
    // takes at most half (1.6 KB a particle), else one without hits (0.2 KB: no
    // more than the checkpoints and adjoints cannot do without, so that a batch
    // that fits at all can be differentiated).  Step and backward of 524,288
    // particles x 16 substeps: 43 ms holding 13.3 GB, 67 ms 1.4 GB, 98 ms 0.7 GB.
    ad_stride = (c + kCoopPad + 63) / 64 * 64;
    const size_t tail = 2 * sizeof(float4) * ad_stride;  // ad_sx0, ad_om
    size_t free_b = 0, total_b = 0;
    ACK(cudaMemGetInfo(&free_b, &total_b));
    for (int kind = 0; kind < 3; ++kind) {
        const bool hits = kind < 2;
        const uint32_t R = kind == 0 ? S : 1u;
        Record probe;
        const size_t bytes = lay_record(*this, probe, nullptr, ad_stride, I, hits);
        if (hits && bytes * R + tail > free_b / (kind == 0 ? 4 : 2)) continue;
        char* slab = nullptr;
        if ((rc = aalloc(slab, bytes * R + (hits ? tail : 0)))) {
            if (hits) continue;
            ad_free();
            return rc;
        }
        ad_slab = slab;
        ad_full = kind == 0;
        records.resize(R);
        for (uint32_t k = 0; k < R; ++k) lay_record(*this, records[k], slab + bytes * k, ad_stride, I, hits);
        ad_sx0 = hits ? reinterpret_cast<float4*>(slab + bytes * R) : sx0;
        ad_om = hits ? ad_sx0 + ad_stride : somega;
        break;
    }
    ad_subs = S;
    ad_iters = I;
    return PBF_OK;
}

// Substep `sub` from (src_pos, src_vel) to (dst_pos, dst_vel), as
// substep_body runs it, with what the reverse passes read kept in r.
int pbf_batch::record_substep(uint32_t sub, Record& r, const float4* src_pos, const float4* src_vel, float4* dst_pos,
                              float4* dst_vel)
{
    const DevParams P = dev_params();
    const int sms = num_sms, G = ad_lanes();
    const uint32_t I = cfg.solver_iterations;
    const bool last = sub + 1 == cfg.substep_iterations;
    float4* x = I ? sx[0] : r.xf;
    if (bcnt) {
        launch_bucket_sort(P, scenes_dev, scene_of, src_pos, src_vel, keys, mka, bcnt, table_size, r.table, mia, r.ids,
                           nullptr, x, r.sv, sx0, lod, sms, stream, &launches);
    } else {
        launch_b_predict(P, scenes_dev, scene_of, src_pos, src_vel, keys, sms, stream);
        launch_radix_sort_into(n, key_bits, keys, ka, r.ids, kb, ib, hist, totals, stream);
        ACK(cudaMemsetAsync(r.table, 0xFF, sizeof(int2) * (size_t)table_size, stream));
        launch_build_table(n, ka, r.table, sms, stream);
        launch_b_reorder(P, scenes_dev, scene_of, r.ids, src_pos, src_vel, x, r.sv, sx0, lod, nullptr, mbits,
                         sms, stream);
        launches += 3 + 3 * ((key_bits + 7) / 8);
    }
    for (uint32_t it = 1; it <= I; ++it) {
        const size_t at = (size_t)(it - 1) * ad_stride;
        float4* xl = r.xl + at;
        uint32_t *list = r.hits(at), *len = r.hit_count(at);
        launch_c_lambda(G, P, scenes_dev, scene_of, sx[0], xl, r.rhol + at, r.table, lod, it, nullptr, list, len,
                        r.auxl + at, stream);
        launch_c_deltap(G, P, scenes_dev, scene_of, xl, it == I ? r.xf : sx[0], r.table, lod, it, nullptr, list, len,
                        r.auxd + at, stream);
        launches += 2;
    }
    float4* x0 = sx0;
    float4* om = somega;
    if (last && cfg.enable_vorticity) {  // the vorticity pass and its reverse read these
        if (ad_sx0 != sx0) ACK(cudaMemcpyAsync(ad_sx0, sx0, sizeof(float4) * n, cudaMemcpyDeviceToDevice, stream));
        x0 = ad_sx0;
        om = ad_om;
    }
    launch_c_integrate(G, P, scenes_dev, scene_of, r.xf, r.sv, x0, om, r.ids, dst_pos, dst_vel, r.table, nullptr,
                       r.hits((size_t)I * ad_stride), r.hit_count((size_t)I * ad_stride), r.fsum, stream);
    ++launches;
    return PBF_OK;
}

int pbf_batch::record_body()
{
    const uint32_t S = cfg.substep_iterations;
    for (uint32_t sub = 0; sub < S; ++sub) {
        ACK(cudaMemcpyAsync(cp_pos + (size_t)sub * n, pos, sizeof(float4) * n, cudaMemcpyDeviceToDevice, stream));
        ACK(cudaMemcpyAsync(cp_vel + (size_t)sub * n, vel, sizeof(float4) * n, cudaMemcpyDeviceToDevice, stream));
        // (a record that the backward fills is not written here)
        const int rc = ad_full ? record_substep(sub, records[sub], pos, vel, pos, vel) : substep_body(pos, vel, pos, vel);
        if (rc) return rc;
    }
    if (cfg.enable_vorticity && !ad_full) {
        vorticity_pass();
    } else if (cfg.enable_vorticity) {
        const Record& r = records[S - 1];
        launch_c_vorticity(ad_lanes(), dev_params(), scenes_dev, scene_of, ad_sx0, ad_om, r.ids, vel, r.table, nullptr,
                           stream);
        ++launches;
    }
    return PBF_OK;
}

// Inputs: pb, vb (adjoints of the recorded step's final state).  Outputs:
// pb, vb (adjoints of its initial state), tgrad (of the SDF translations).
int pbf_batch::backward_body(bool recompute)
{
    const DevParams P = dev_params();
    const int sms = num_sms, G = ad_lanes();
    const uint32_t S = cfg.substep_iterations, I = cfg.solver_iterations;
    const bool vort = cfg.enable_vorticity != 0;
    ACK(cudaMemsetAsync(tgrad, 0, sizeof(float) * 4 * scenes.size(), stream));
    ACK(cudaMemsetAsync(pbs, 0, sizeof(float4) * n, stream));
    ACK(cudaMemsetAsync(omb, 0, sizeof(float4) * n, stream));
    // accumulated with atomics; each pass that is through with one clears it
    ACK(cudaMemsetAsync(gxa, 0, sizeof(float4) * n, stream));
    ACK(cudaMemsetAsync(gxb, 0, sizeof(float4) * n, stream));
    ACK(cudaMemsetAsync(gv, 0, sizeof(float4) * n, stream));
    float4 *a = gxa, *b = gxb;
    for (int sub = (int)S - 1; sub >= 0; --sub) {
        const float4* src_pos = cp_pos + (size_t)sub * n;
        const float4* src_vel = cp_vel + (size_t)sub * n;
        Record& r = records[ad_full ? sub : 0];
        if (recompute) {
            const int rc = record_substep((uint32_t)sub, r, src_pos, src_vel, tpos, tvel);
            if (rc) return rc;
        }
        const bool last = (sub == (int)S - 1) && vort;
        if (last) {
            launch_ac_vorticity(G, P, scenes_dev, scene_of, r.table, ad_sx0, ad_om, r.ids, vb, pbs, omb, stream);
            ++launches;
        }
        launch_ac_integrate(G, P, scenes_dev, scene_of, r.table, r.hits((size_t)I * ad_stride),
                            r.hit_count((size_t)I * ad_stride), r.fsum, r.xf, r.sv, src_pos, r.ids, pb, vb,
                            last ? pbs : nullptr, last ? omb : nullptr, ad_om, a, gv, x0b, tgrad, stream);
        ++launches;
        for (int it = (int)I; it >= 1; --it) {
            const size_t at = (size_t)(it - 1) * ad_stride;
            const uint32_t *list = r.hits(at), *len = r.hit_count(at);
            launch_ac_deltap(G, P, scenes_dev, scene_of, r.table, list, len, r.xl + at, r.auxd + at, a, b, tgrad, stream);
            launch_ac_lambda(G, P, scenes_dev, scene_of, r.table, list, len, r.xl + at, r.auxl + at, r.rhol + at, b, a,
                             stream);
            launches += 2;
            std::swap(a, b);
        }
        launch_ad_predict(n, P.dt, r.ids, a, gv, x0b, pb, vb, sms, stream);
        ++launches;
    }
    return PBF_OK;
}

// Run body() once, through a graph captured on first use when enabled.
template <class Body>
static int run_graph(pbf_batch* b, cudaGraph_t& g, cudaGraphExec_t& ex, uint64_t& glaunches, Body body)
{
    if (!b->use_graph) return body();
    if (!ex) {
        const uint64_t before = b->launches;
        b->capturing = true;
        ACK(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
        const int rc = body();
        cudaGraph_t gg = nullptr;
        const cudaError_t e = cudaStreamEndCapture(b->stream, &gg);
        b->capturing = false;
        if (rc) {
            if (gg) cudaGraphDestroy(gg);
            return rc;
        }
        if (e != cudaSuccess) return set_error(PBF_ERR_CUDA, "cudaStreamEndCapture: %s", cudaGetErrorString(e));
        g = gg;
        ACK(cudaGraphInstantiate(&ex, g, 0));
        glaunches = b->launches - before;
        b->launches = before;
    }
    ACK(cudaGraphLaunch(ex, b->stream));
    b->launches += glaunches;
    return PBF_OK;
}

static int check_differentiable(const pbf_batch* b)
{
    if (b->cfg.enable_apbf) return set_error(PBF_ERR_STATE, "the adjoint needs APBF off");
    if (b->n == 0) return set_error(PBF_ERR_STATE, "empty batch");
    return PBF_OK;
}

// ---- C ABI --------------------------------------------------------------------------------
#define CHECK_B(b)                                                                                 \
    do {                                                                                           \
        if (!(b)) return pbf::set_error(PBF_ERR_INVALID, "null batch");                            \
        cudaError_t e_ = cudaSetDevice((b)->device);                                               \
        if (e_ != cudaSuccess)                                                                     \
            return pbf::set_error(PBF_ERR_CUDA, "cudaSetDevice: %s", cudaGetErrorString(e_));      \
    } while (0)

extern "C" int pbf_batch_set_sdf_offset(pbf_batch* b, uint32_t scene, const float t[3])
{
    CHECK_B(b);
    if (scene >= b->scenes.size()) return set_error(PBF_ERR_INVALID, "scene %u out of range", scene);
    if (!t) return set_error(PBF_ERR_INVALID, "null offset");
    for (int a = 0; a < 3; ++a) b->scenes[scene].sdf_offset[a] = t[a];
    b->recorded = false;
    return b->upload_scenes();
}

extern "C" int pbf_batch_set_state(pbf_batch* b, const void* pos4, const void* vel4)
{
    CHECK_B(b);
    if (b->n == 0) return PBF_OK;
    if (!pos4 || !vel4) return set_error(PBF_ERR_INVALID, "null state");
    ACK(cudaMemcpyAsync(b->pos, pos4, sizeof(float4) * b->n, cudaMemcpyDefault, b->stream));
    ACK(cudaMemcpyAsync(b->vel, vel4, sizeof(float4) * b->n, cudaMemcpyDefault, b->stream));
    ACK(cudaStreamSynchronize(b->stream));
    b->recorded = false;
    return PBF_OK;
}

extern "C" int pbf_batch_get_state(pbf_batch* b, void* pos4, void* vel4)
{
    CHECK_B(b);
    if (b->n == 0) return PBF_OK;
    if (pos4) ACK(cudaMemcpyAsync(pos4, b->pos, sizeof(float4) * b->n, cudaMemcpyDefault, b->stream));
    if (vel4) ACK(cudaMemcpyAsync(vel4, b->vel, sizeof(float4) * b->n, cudaMemcpyDefault, b->stream));
    ACK(cudaStreamSynchronize(b->stream));
    return PBF_OK;
}

extern "C" int pbf_batch_forward_record(pbf_batch* b)
{
    CHECK_B(b);
    int rc = check_differentiable(b);
    if (rc) return rc;
    if ((rc = b->ad_alloc())) return rc;
    rc = run_graph(b, b->rec_graph, b->rec_exec, b->rec_launches, [&] { return b->record_body(); });
    if (rc) return rc;
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return set_error(PBF_ERR_CUDA, "kernel launch: %s", cudaGetErrorString(e));
    b->recorded = true;
    b->recorded_gen = b->scenes_gen;
    return PBF_OK;
}

extern "C" int pbf_batch_backward(pbf_batch* b, const void* gpos4, const void* gvel4, void* out_gpos4,
                                  void* out_gvel4, float* out_gt)
{
    CHECK_B(b);
    int rc = check_differentiable(b);
    if (rc) return rc;
    if (!b->recorded) return set_error(PBF_ERR_STATE, "backward without a recorded forward");
    const size_t bytes = sizeof(float4) * b->n;
    if (gpos4) ACK(cudaMemcpyAsync(b->pb, gpos4, bytes, cudaMemcpyDefault, b->stream));
    else ACK(cudaMemsetAsync(b->pb, 0, bytes, b->stream));
    if (gvel4) ACK(cudaMemcpyAsync(b->vb, gvel4, bytes, cudaMemcpyDefault, b->stream));
    else ACK(cudaMemsetAsync(b->vb, 0, bytes, b->stream));
    // the records hold for the scenes they were made under
    const bool recompute = !b->ad_full || b->recorded_gen != b->scenes_gen;
    if (b->bwd_exec && b->bwd_recompute != recompute) {
        cudaGraphExecDestroy(b->bwd_exec);
        cudaGraphDestroy(b->bwd_graph);
        b->bwd_exec = nullptr;
        b->bwd_graph = nullptr;
    }
    b->bwd_recompute = recompute;
    rc = run_graph(b, b->bwd_graph, b->bwd_exec, b->bwd_launches, [&] { return b->backward_body(recompute); });
    if (rc) return rc;
    if (out_gpos4) ACK(cudaMemcpyAsync(out_gpos4, b->pb, bytes, cudaMemcpyDefault, b->stream));
    if (out_gvel4) ACK(cudaMemcpyAsync(out_gvel4, b->vb, bytes, cudaMemcpyDefault, b->stream));
    if (out_gt) {
        std::vector<float> t(4 * b->scenes.size());
        ACK(cudaMemcpyAsync(t.data(), b->tgrad, sizeof(float) * t.size(), cudaMemcpyDeviceToHost, b->stream));
        ACK(cudaStreamSynchronize(b->stream));
        for (size_t k = 0; k < b->scenes.size(); ++k)
            for (int a = 0; a < 3; ++a) out_gt[3 * k + a] = t[4 * k + a];
    }
    ACK(cudaStreamSynchronize(b->stream));
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return set_error(PBF_ERR_CUDA, "kernel launch: %s", cudaGetErrorString(e));
    return PBF_OK;
}
