// Incremental generation: one token per sequence and call, with the bit
// histories of every (sequence, layer, channel) kept on the device between
// calls (reference UllisHeron::generate_state / generate_step, src/model.rs:2691-2753;
// per-block forward_one src/model.rs:2243-2262, ROSA 1320-1352, CMix 1003-1016).
//
// A step is a handful of [batch, d_model] row operations, so it runs on the
// CUDA cores in the reference's summation order: the logits of step t
// are bit-identical to row t of the one-shot forward in EXACT mode, which is
// what the reference's own test asserts (src/model.rs:4991-5004).  The whole
// step is one kernel of thread-block clusters (generate_step.cuh) where the
// shape allows; otherwise its ~90 small launches are replayed as one CUDA graph
// (two graphs: before and after the first token, which has no time-shift
// history).
// A stream's automaton is not kept: a push is answered from the bit histories
// (gen_push.cuh).
#include "generate.hpp"

#include <cuda_fp16.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "generate_plan.hpp"
#include "generate_step.cuh"
#include "kernels.hpp"
#include "linear_tc.hpp"

namespace ullis {
namespace {

inline unsigned blocks_for(size_t n, unsigned per) { return (unsigned)((n + per - 1) / per); }

__device__ __forceinline__ float h2f(uint16_t b) { return __half2float(__ushort_as_half(b)); }

// time_shift_one + mixes (src/model.rs:214-228, 1331-1340, 1008-1012): xx = prev - x, or -x before the
// first token; out_m = x + xx*mix_m, unfused; then x becomes the layer's new time-shift history
__global__ void gen_shift_mix_kernel(const float* __restrict__ x, float* __restrict__ prev, int has_prev,
                                     const uint16_t* __restrict__ m0, const uint16_t* __restrict__ m1,
                                     const uint16_t* __restrict__ m2, float* __restrict__ o0, float* __restrict__ o1,
                                     float* __restrict__ o2, size_t n, size_t C) {
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    const size_t c = e % C;
    const float xt = x[e];
    const float xx = has_prev ? __fsub_rn(prev[e], xt) : -xt;
    o0[e] = __fadd_rn(xt, __fmul_rn(xx, h2f(m0[c])));
    if (o1) o1[e] = __fadd_rn(xt, __fmul_rn(xx, h2f(m1[c])));
    if (o2) o2[e] = __fadd_rn(xt, __fmul_rn(xx, h2f(m2[c])));
    prev[e] = xt;
}

// LayerNorm of one row and the time-shift mixes of that row in one launch (the two kernels above it in a step,
// for the few rows of a step): the reference's LayerNorm arithmetic (src/model.rs:259-276: the sum, then the sum
// of the squared deviations, each added one value after the other) is a chain one thread has to run, 2·C
// dependent additions; it runs from shared memory, and the rest of the CTA does the affine part, the mixes and
// the new time-shift history.  `ln_out` (nullable) receives the normalised row.
__global__ void __launch_bounds__(128)
gen_ln_shift_mix_kernel(const float* __restrict__ x, const uint16_t* __restrict__ lw, const uint16_t* __restrict__ lb,
                        float* __restrict__ ln_out, float* __restrict__ prev, int has_prev,
                        const uint16_t* __restrict__ m0, const uint16_t* __restrict__ m1,
                        const uint16_t* __restrict__ m2, float* __restrict__ o0, float* __restrict__ o1,
                        float* __restrict__ o2, size_t C) {
    extern __shared__ __align__(16) float gen_row[];
    __shared__ float s_mean, s_inv;
    const size_t r = blockIdx.x;
    for (size_t c = threadIdx.x; c < C; c += blockDim.x) gen_row[c] = x[r * C + c];
    __syncthreads();
    if (threadIdx.x == 0) {
        // the additions are one chain; the loads are not: sixteen values are fetched (four 16-byte loads) before
        // they are added, so that the chain waits for arithmetic only
        float acc = 0.0f;
        size_t c = 0;
        for (; c + 16 <= C; c += 16) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = *reinterpret_cast<const float4*>(gen_row + c + 4 * u);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                acc = __fadd_rn(acc, v[u].x); acc = __fadd_rn(acc, v[u].y);
                acc = __fadd_rn(acc, v[u].z); acc = __fadd_rn(acc, v[u].w);
            }
        }
        for (; c < C; ++c) acc = __fadd_rn(acc, gen_row[c]);
        const float mean = __fdiv_rn(acc, (float)C);
        acc = 0.0f;
        for (c = 0; c + 16 <= C; c += 16) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = *reinterpret_cast<const float4*>(gen_row + c + 4 * u);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float d0 = __fsub_rn(v[u].x, mean), d1 = __fsub_rn(v[u].y, mean);
                const float d2 = __fsub_rn(v[u].z, mean), d3 = __fsub_rn(v[u].w, mean);
                acc = __fadd_rn(acc, __fmul_rn(d0, d0)); acc = __fadd_rn(acc, __fmul_rn(d1, d1));
                acc = __fadd_rn(acc, __fmul_rn(d2, d2)); acc = __fadd_rn(acc, __fmul_rn(d3, d3));
            }
        }
        for (; c < C; ++c) {
            const float dlt = __fsub_rn(gen_row[c], mean);
            acc = __fadd_rn(acc, __fmul_rn(dlt, dlt));
        }
        s_mean = mean;
        s_inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(acc, (float)C), 1e-5f)));
    }
    __syncthreads();
    const float mean = s_mean, inv = s_inv;
    for (size_t c = threadIdx.x; c < C; c += blockDim.x) {
        const size_t e = r * C + c;
        const float n = __fmul_rn(__fsub_rn(gen_row[c], mean), inv);
        const float xt = __fadd_rn(__fmul_rn(n, h2f(lw[c])), h2f(lb[c]));
        if (ln_out) ln_out[e] = xt;
        // time_shift_one + mixes (src/model.rs:214-228, 1331-1340, 1008-1012), as gen_shift_mix_kernel
        const float xx = has_prev ? __fsub_rn(prev[e], xt) : -xt;
        o0[e] = __fadd_rn(xt, __fmul_rn(xx, h2f(m0[c])));
        if (o1) o1[e] = __fadd_rn(xt, __fmul_rn(xx, h2f(m1[c])));
        if (o2) o2[e] = __fadd_rn(xt, __fmul_rn(xx, h2f(m2[c])));
        prev[e] = xt;
    }
}

// one RosaSam::push per (sequence, channel) of one layer and y = (2*idx - 1)*e (src/model.rs:1344-1351); `per_warp`
// streams per warp
__global__ void __launch_bounds__(128)
gen_push_kernel(push::Histories H, size_t first, const uint32_t* __restrict__ time, uint32_t per_warp, const float* __restrict__ q,
                const float* __restrict__ k, const float* __restrict__ v, const uint16_t* __restrict__ e, float* __restrict__ y,
                size_t streams, size_t C) {
    const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, s = warp * per_warp + (threadIdx.x & 31u);
    const bool live = (threadIdx.x & 31u) < per_warp && s < streams;
    // src/rosa.rs:372-374: bit = activation > 0
    const size_t f = first + warp * per_warp;
    const uint32_t i = *time;
    const bool idx = push::step(H, f, live, i, push::begin(H, f, live, i), live && q[s] > 0.0f, live && k[s] > 0.0f, live && v[s] > 0.0f);
    if (live) {
        const float ev = h2f(e[s % C]);
        y[s] = idx ? ev : -ev;
    }
}

// `steps` pushes of every stream, bits as bytes [steps, streams]
__global__ void __launch_bounds__(128)
push_steps_kernel(push::Histories H, size_t time, size_t steps, uint32_t per_warp, const uint8_t* __restrict__ q,
                  const uint8_t* __restrict__ k, const uint8_t* __restrict__ v, uint8_t* __restrict__ idx, size_t streams) {
    const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, s = warp * per_warp + (threadIdx.x & 31u);
    const bool live = (threadIdx.x & 31u) < per_warp && s < streams;
    for (size_t t = 0; t < steps; ++t) {
        const size_t at = t * streams + s;
        const size_t f = warp * per_warp;
        const uint32_t i = (uint32_t)(time + t);
        const bool bit = push::step(H, f, live, i, push::begin(H, f, live, i), live && q[at], live && k[at], live && v[at]);
        if (live) idx[at] = bit;
        __syncwarp();   // a lane's words are read by the whole warp in the next step
    }
}

// Streams per warp: a warp takes its streams' searches one after the other, so no more than keep the device busy.
uint32_t streams_per_warp(const ullis_cuda_runtime* rt, size_t streams) {
    uint32_t n = 1;
    while (n < 32u && streams > (size_t)n * (size_t)rt->sm_count * 32u) n *= 2;
    return n;
}

}  // namespace
}  // namespace ullis

using namespace ullis;

ullis_cuda_generate_state::ullis_cuda_generate_state(ullis_cuda_model* m, size_t batch_) : model(m), batch(batch_) {
    if (batch == 0) fail(ULLIS_CUDA_ERR_SHAPE, "generate needs at least one sequence");
    wps = (m->context_len + 31) / 32;
    const size_t per_layer = batch * m->d;
    if (per_layer / m->d != batch || m->layers > SIZE_MAX / per_layer) fail(ULLIS_CUDA_ERR_SHAPE, "generate state shape overflow");
    streams = m->layers * per_layer;
    if (streams > SIZE_MAX / (wps * 12 + sizeof(push::Current))) fail(ULLIS_CUDA_ERR_SHAPE, "generate state shape overflow");
    ullis_cuda_runtime* rt = m->rt;
    rt->bind();
    k::rowvec_prepare(rt);   // before any step is recorded into a graph
    words.ensure(streams * wps * 12);
    current.ensure(streams * sizeof(push::Current));
    prev.ensure(2 * m->layers * 2 * per_layer * 4);   // read one half, write the other (generate_step.cuh)
    ids.ensure((batch + 1) * 4);
    for (ullis::DeviceBuffer* buf : {&x, &a, &bq, &bk, &bv}) buf->ensure(per_layer * 4);
    wide.ensure(batch * std::max(m->ffn, 3 * m->d) * 4);
    logits.ensure(batch * m->vocab * 4);
    ULLIS_CUDA_CHECK(cudaMallocHost(&h_tokens, (batch + 1) * 4));
    ULLIS_CUDA_CHECK(cudaMallocHost(&h_logits, batch * m->vocab * 4));
    use_graph = !getenv("ULLIS_CUDA_NO_GRAPH");
    if (const char* env = getenv("ULLIS_CUDA_INJECT_GENERATE_FAILURE")) inject_failure_at = (size_t)std::max(0, atoi(env));
    if (const char* env = getenv("ULLIS_CUDA_GEN_WAIT_POLLS")) wait_polls = (uint32_t)std::min(std::max(0, atoi(env)), 1 << 18);
    prepare_one_kernel();
    reset();
}

// Whether a step of this shape runs as one kernel, and how it is split over clusters.
void ullis_cuda_generate_state::prepare_one_kernel() {
    ullis_cuda_model* m = model;
    ullis_cuda_runtime* rt = m->rt;
    if (getenv("ULLIS_CUDA_GEN_UNFUSED") || getenv("ULLIS_CUDA_NO_GRAPH") || m->d % 32 || m->ffn % gen::PIECE || rt->cc_major < 9) return;
    auto kernel_for = [](uint32_t g, uint32_t own) {
        const gen::StepShape shape = gen::step_shape(g, own);
        if (g == 1) return reinterpret_cast<const void*>(gen::gen_step_kernel<1, gen::PLAIN>);
#define ULLIS_STEP_OF(G)                                                                                     \
    (shape == gen::BY_ROW ? reinterpret_cast<const void*>(gen::gen_step_kernel<G, gen::BY_ROW>)              \
     : shape == gen::WIDE ? reinterpret_cast<const void*>(gen::gen_step_kernel<G, gen::WIDE>)                \
                          : reinterpret_cast<const void*>(gen::gen_step_kernel<G, gen::PLAIN>))
        return g == 2 ? ULLIS_STEP_OF(2) : ULLIS_STEP_OF(4);
#undef ULLIS_STEP_OF
    };
    constexpr size_t MOST_SMEM = 224 * 1024;
    const auto prepare = [&](const void* kernel) {
        ULLIS_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MOST_SMEM));
        ULLIS_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    };
    const auto room = [&](const void* kernel, const gen::StepPlan& p) {
        cudaLaunchAttribute attr;
        const cudaLaunchConfig_t cfg = step_config(&attr, p.cluster, p.cluster, p.smem);
        int clusters = 0;
        ULLIS_CUDA_CHECK(cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg));
        return clusters;
    };
    const uint32_t d = (uint32_t)m->d, ffn = (uint32_t)m->ffn;
    const auto fit = [&](gen::StepPlan& p) {   // packed weights stay where they are if there is no room for them beside the ring
        for (const bool staged : {true, false}) {
            p.staged = staged;
            p.stages = gen::ring_stages(p.group, d, ffn, p.cluster, staged, MOST_SMEM);
            p.smem = gen::Layout(p.group, d, ffn, p.cluster, p.stages, staged).total;
            if (p.smem <= MOST_SMEM) break;
        }
        return p.smem <= MOST_SMEM && p.stages <= gen::MAX_STAGES;
    };
    // An SM holds one CTA of any form, by its registers, so any of them tells how much room there is (a form is loaded when it is asked for, 3 ms
    // each, and the question takes 0.1 ms more); the one that is taken is asked where that does not hold.
    const auto alone = [&](const void* kernel) {
        cudaFuncAttributes attr;
        ULLIS_CUDA_CHECK(cudaFuncGetAttributes(&attr, kernel));
        return (size_t)attr.numRegs * gen::THREADS * 2 > 64 * 1024;
    };
    const void* any_form = kernel_for(1, 32);
    prepare(any_form);
    const gen::StepPlan plan = gen::plan_step(
        batch, gen::MAX_CLUSTER, gen::MAX_GROUP, [&](uint32_t c) { return d % (c * 32) == 0 && ffn % (c * 4) == 0; }, fit,
        [&](const gen::StepPlan& p) { return room(any_form, p); },
        [&](const gen::StepPlan& p) {
            step_kernel = kernel_for(p.group, d / p.cluster);
            prepare(step_kernel);
            return alone(any_form) && alone(step_kernel) ? p.clusters : room(step_kernel, p);
        });
    if (!plan.grid) return;
    cluster = plan.cluster; group = plan.group; step_stages = plan.stages; step_staged = plan.staged; step_smem = plan.smem; step_grid = plan.grid;
    std::vector<gen::Layer> layers(m->layers);
    for (size_t l = 0; l < m->layers; ++l) {
        const LayerWeights& L = m->blocks[l];
        auto packed = [](const PackedWeights& w) { return gen::Packed{w.bits, w.scale, w.bias}; };
        layers[l] = gen::Layer{L.ln3.weight, L.ln3.bias, {L.x_q, L.x_k, L.x_v}, L.e, L.ln2.weight, L.ln2.bias, L.ffn_x_k,
                               {packed(L.q), packed(L.k), packed(L.v)}, packed(L.o), gen::Packed{L.key.bits, L.key.scale, nullptr}};
    }
    std::vector<CUtensorMap> values;
    const uint32_t own = (uint32_t)m->d / cluster, slabs = group * own == gen::VALUE_OUT ? (uint32_t)m->ffn / gen::SLAB : own <= gen::MAX_BOX ? gen::PIECE / gen::SLAB : 1u;
    for (size_t l = 0; l < m->layers; ++l) values.push_back(tc::slab_map(m->blocks[l].value, m->d, m->ffn, std::min(own, gen::MAX_BOX), slabs));
    step_layers.ensure(layers.size() * sizeof(gen::Layer) + 16);
    step_values.ensure(values.size() * sizeof(CUtensorMap));
    rt->h2d(step_layers.get(), layers.data(), layers.size() * sizeof(gen::Layer));
    rt->h2d(step_values.get(), values.data(), values.size() * sizeof(CUtensorMap));
    rt->sync();
}

cudaLaunchConfig_t ullis_cuda_generate_state::step_config(cudaLaunchAttribute* attr, unsigned grid, unsigned per_cluster, size_t smem) const {
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = per_cluster;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(gen::THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = model->rt->stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

ullis_cuda_generate_state::~ullis_cuda_generate_state() {
    for (cudaGraphExec_t g : graph)
        if (g) cudaGraphExecDestroy(g);
    if (h_tokens) cudaFreeHost(h_tokens);
    if (h_logits) cudaFreeHost(h_logits);
}

// Empty histories (src/rosa.rs:66-74): a push at position 0 looks at nothing that was there before.
void ullis_cuda_generate_state::reset() {
    ullis_cuda_runtime* rt = model->rt;
    rt->bind();
    if (poisoned) rt->sync();   // whatever failed has left the device before the next step starts
    time = 0;
    poisoned = false;
}

ullis::push::Histories ullis_cuda_generate_state::histories() {
    return {static_cast<push::Current*>(current.get()), static_cast<uint32_t*>(words.get()), wps};
}

// Enqueues a step as one kernel; logits_to: device memory or page-locked host memory.
void ullis_cuda_generate_state::launch_one_kernel(float* logits_to) {
    ullis_cuda_model* m = model;
    ullis_cuda_runtime* rt = m->rt;
    const size_t half = m->layers * 2 * batch * m->d;
    float* history = static_cast<float*>(prev.get());
    gen::Step p{};
    p.layers = static_cast<const gen::Layer*>(step_layers.get());
    p.values = static_cast<const CUtensorMap*>(step_values.get());
    p.staged = step_staged;
    p.polls = wait_polls;
    p.status = rt->host_status;
    p.n_layers = (uint32_t)m->layers; p.rows = (uint32_t)batch; p.d = (uint32_t)m->d; p.ffn = (uint32_t)m->ffn;
    p.vocab = (uint32_t)m->vocab; p.time = (uint32_t)time;
    p.stages = step_stages;
    p.minus_zero = -0.0f;
    p.tokens = h_tokens;
    p.embedding = m->embedding;
    p.ln0_w = m->blocks[0].ln0.weight; p.ln0_b = m->blocks[0].ln0.bias;
    p.ln_out_w = m->ln_out.weight; p.ln_out_b = m->ln_out.bias;
    p.head = gen::Packed{m->head.bits, m->head.scale, m->head.bias};
    p.prev_in = history + (time & 1) * half;
    p.prev_out = history + (~time & 1) * half;
    p.push = histories();
    p.logits = logits_to;
    rt->host_status[0] = ULLIS_DEV_OK;   // the kernel writes there itself
    void* args[] = {&p};
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = step_config(&attr, step_grid, cluster, step_smem);
    ULLIS_CUDA_CHECK(cudaLaunchKernelExC(&cfg, step_kernel, args));
    rt->launched("gen_step");
}

void ullis_cuda_generate_state::step(const uint32_t* tokens, float* logits_out) {
    ullis_cuda_model* m = model;
    ullis_cuda_runtime* rt = m->rt;
    // src/model.rs:2718-2723
    for (size_t b = 0; b < batch; ++b)
        if (tokens[b] >= m->vocab) fail(ULLIS_CUDA_ERR_TOKEN, "token id exceeds vocabulary");
    if (time >= m->context_len)
        fail(ULLIS_CUDA_ERR_SHAPE, "generate exceeded context_len (" + std::to_string(m->context_len) + ")");
    if (poisoned)
        fail(ULLIS_CUDA_ERR_ARG, "generate state is unusable after a failed step: reset it (ullis_cuda_generate_state_reset)");
    rt->bind();
    if (rt->kernel_timing) rt->mark("(between steps)");
    std::memcpy(h_tokens, tokens, batch * 4);
    h_tokens[batch] = (uint32_t)time;
    const int has_prev = time != 0;
    // From here on the device-side histories and time-shift inputs may have moved on by one position
    // while `time` has not: a failure below leaves the state out of step with itself, and a retry would push the
    // same position twice.  The state stays refused until reset() (which rebuilds it from scratch).
    struct Poison {
        bool* flag;
        bool armed = true;
        ~Poison() { if (armed) *flag = true; }
    } poison{&poisoned};

    // The logits go straight into page-locked memory (what the Python layer passes), else through h_logits.
    float* to = logits_out;
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, logits_out) != cudaSuccess || attr.type != cudaMemoryTypeHost) {
        cudaGetLastError();
        to = h_logits;
    }
    if (step_grid) {
        if (batch <= DIRECT_LOGITS) {
            launch_one_kernel(to);
        } else {
            launch_one_kernel(static_cast<float*>(logits.get()));
            rt->d2h(to, logits.get(), batch * m->vocab * 4);
        }
    } else if (use_graph && !rt->kernel_timing) {
        // Replay the step as one graph launch; per-kernel timing needs the plain launches.
        if (!graph[has_prev]) {
            cudaGraph_t captured = nullptr;
            const uint64_t before = rt->launches;
            ULLIS_CUDA_CHECK(cudaStreamBeginCapture(rt->stream, cudaStreamCaptureModeThreadLocal));
            try {
                enqueue(has_prev);
            } catch (...) {
                cudaStreamEndCapture(rt->stream, &captured);
                if (captured) cudaGraphDestroy(captured);
                rt->launches = before;
                throw;
            }
            ULLIS_CUDA_CHECK(cudaStreamEndCapture(rt->stream, &captured));
            graph_launches = rt->launches - before;
            rt->launches = before;   // counted per replay below
            const cudaError_t e = cudaGraphInstantiate(&graph[has_prev], captured, 0);
            cudaGraphDestroy(captured);
            ULLIS_CUDA_CHECK(e);
        }
        ULLIS_CUDA_CHECK(cudaGraphLaunch(graph[has_prev], rt->stream));
        rt->launches += graph_launches;
        to = h_logits;
    } else {
        enqueue(has_prev);
        to = h_logits;
    }
    rt->sync();
    rt->throw_on_status();
    if (inject_failure_at && time + 1 == inject_failure_at) {   // host-injected: what a CUDA error after the launches does
        inject_failure_at = 0;
        fail(ULLIS_CUDA_ERR_CUDA, "injected failure after the step's kernels ran");
    }
    if (to != logits_out) std::memcpy(logits_out, to, batch * m->vocab * 4);
    time += 1;
    poison.armed = false;
}

void ullis_cuda_generate_state::enqueue(int has_prev) {
    ullis_cuda_model* m = model;
    ullis_cuda_runtime* rt = m->rt;
    const size_t d = m->d, ffn = m->ffn, rows = batch, n = rows * d;
    uint32_t* IDS = static_cast<uint32_t*>(ids.get());
    float* X = static_cast<float*>(x.get());
    float* A = static_cast<float*>(a.get());
    float* Bq = static_cast<float*>(bq.get());
    float* Bk = static_cast<float*>(bk.get());
    float* Bv = static_cast<float*>(bv.get());
    float* W = static_cast<float*>(wide.get());
    float* LG = static_cast<float*>(logits.get());
    rt->clear_status();
    rt->h2d(IDS, h_tokens, (rows + 1) * 4);   // the ids and the position: a recorded graph takes both from here
    k::embed(rt, IDS, m->embedding, X, rows, d, m->vocab);
    const bool fused_ln = d * 4 <= 48 * 1024 && !getenv("ULLIS_CUDA_GEN_UNFUSED");   // a row in shared memory
    for (size_t l = 0; l < m->layers; ++l) {
        const LayerWeights& L = m->blocks[l];
        float* rosa_prev = static_cast<float*>(prev.get()) + (l * 2) * n;
        float* cmix_prev = rosa_prev + n;
        const size_t s0 = l * n;  // first stream of this layer
        if (l == 0) {  // ln0 REPLACES x on layer 0 (src/model.rs:2244-2248)
            k::layer_norm(rt, X, L.ln0.weight, L.ln0.bias, A, rows, d, true);
            ULLIS_CUDA_CHECK(cudaMemcpyAsync(X, A, n * 4, cudaMemcpyDeviceToDevice, rt->stream));
        }
        // ROSA (src/model.rs:1320-1352)
        if (fused_ln) {
            gen_ln_shift_mix_kernel<<<(unsigned)rows, 128, d * 4, rt->stream>>>(X, L.ln3.weight, L.ln3.bias, nullptr, rosa_prev,
                                                                                has_prev, L.x_q, L.x_k, L.x_v, Bq, Bk, Bv, d);
            rt->launched("gen_ln_shift_mix");
        } else {
            k::layer_norm(rt, X, L.ln3.weight, L.ln3.bias, A, rows, d, true);
            gen_shift_mix_kernel<<<blocks_for(n, 256), 256, 0, rt->stream>>>(A, rosa_prev, has_prev, L.x_q, L.x_k, L.x_v, Bq,
                                                                           Bk, Bv, n, d);
            rt->launched("gen_shift_mix");
        }
        {   // Q, K and V in one launch when the shape allows
            const float* xs[3] = {Bq, Bk, Bv};
            const uint32_t* bs[3] = {L.q.bits, L.k.bits, L.v.bits};
            const uint16_t* ss[3] = {L.q.scale, L.k.scale, L.v.scale};
            const uint16_t* bi[3] = {L.q.bias, L.k.bias, L.v.bias};
            float* ys[3] = {W, W + n, W + 2 * n};
            if (!fused_ln || !k::binary_rowvec_multi(rt, 3, xs, bs, ss, bi, ys, rows, d, d, false)) {
                k::binary_linear_exact(rt, Bq, L.q.bits, L.q.scale, L.q.bias, W, rows, d, d, false);
                k::binary_linear_exact(rt, Bk, L.k.bits, L.k.scale, L.k.bias, W + n, rows, d, d, false);
                k::binary_linear_exact(rt, Bv, L.v.bits, L.v.scale, L.v.bias, W + 2 * n, rows, d, d, false);
            }
        }
        {
            const uint32_t per = streams_per_warp(rt, n);
            gen_push_kernel<<<blocks_for((n + per - 1) / per * 32, 128), 128, 0, rt->stream>>>(
                histories(), s0, IDS + batch, per, W, W + n, W + 2 * n, L.e, A, n, d);
            rt->launched("gen_push");
        }
        k::binary_linear_exact(rt, A, L.o.bits, L.o.scale, L.o.bias, X, rows, d, d, true);  // h += rosa out
        // CMix (src/model.rs:1003-1016)
        if (fused_ln) {
            gen_ln_shift_mix_kernel<<<(unsigned)rows, 128, d * 4, rt->stream>>>(X, L.ln2.weight, L.ln2.bias, nullptr, cmix_prev,
                                                                                has_prev, L.ffn_x_k, nullptr, nullptr, Bq, nullptr,
                                                                                nullptr, d);
            rt->launched("gen_ln_shift_mix");
        } else {
            k::layer_norm(rt, X, L.ln2.weight, L.ln2.bias, A, rows, d, true);
            gen_shift_mix_kernel<<<blocks_for(n, 256), 256, 0, rt->stream>>>(A, cmix_prev, has_prev, L.ffn_x_k, nullptr, nullptr,
                                                                           Bq, nullptr, nullptr, n, d);
            rt->launched("gen_shift_mix");
        }
        {   // key and relu^2 in one launch when the shape allows
            const float* xs[1] = {Bq};
            const uint32_t* bs[1] = {L.key.bits};
            const uint16_t* ss[1] = {L.key.scale};
            const uint16_t* bi[1] = {nullptr};
            float* ys[1] = {W};
            if (!fused_ln || !k::binary_rowvec_multi(rt, 1, xs, bs, ss, bi, ys, rows, d, ffn, true)) {
                k::binary_linear_exact(rt, Bq, L.key.bits, L.key.scale, nullptr, W, rows, d, ffn, false);
                k::relu2(rt, W, W, rows * ffn);
            }
        }
        k::fp16_linear_exact(rt, W, L.value, X, rows, ffn, d, true);  // h += cmix out
    }
    // src/model.rs:2750-2752
    k::layer_norm(rt, X, m->ln_out.weight, m->ln_out.bias, A, rows, d, true);
    k::binary_linear_exact(rt, A, m->head.bits, m->head.scale, m->head.bias, LG, rows, d, m->vocab, false);
    rt->d2h(h_logits, LG, rows * m->vocab * 4);
    rt->d2h(rt->host_status, rt->dev_status, 16);
}

// ------------------------------------------------------------------ op level: RosaSam::push for many streams

ullis_cuda_rosa_pushers::ullis_cuda_rosa_pushers(ullis_cuda_runtime* rt_, size_t streams_, size_t capacity_)
    : rt(rt_), streams(streams_), capacity(capacity_) {
    if (streams == 0 || capacity == 0) fail(ULLIS_CUDA_ERR_SHAPE, "ROSA pushers need at least one stream and one position");
    if (capacity > 0x7FFFFFF0u) fail(ULLIS_CUDA_ERR_SHAPE, "ROSA pushers: capacity too large");
    wps = (capacity + 31) / 32;
    if (streams > SIZE_MAX / (wps * 12 + sizeof(push::Current))) fail(ULLIS_CUDA_ERR_SHAPE, "ROSA pushers: shape overflow");
    rt->bind();
    words.ensure(streams * wps * 12);
    current.ensure(streams * sizeof(push::Current));
}

void ullis_cuda_rosa_pushers::reset() { time = 0; }   // a push at position 0 looks at nothing that was there before

void ullis_cuda_rosa_pushers::push(const uint8_t* q, const uint8_t* k, const uint8_t* v, size_t steps, uint8_t* idx) {
    // RosaSam has no capacity (src/rosa.rs:55-64 grows its vectors); here it is fixed when the state is made
    if (steps > capacity - time) fail(ULLIS_CUDA_ERR_SHAPE, "ROSA pushers: more pushes than the capacity given at creation");
    if (steps == 0) return;
    if (steps > SIZE_MAX / streams / 20) fail(ULLIS_CUDA_ERR_SHAPE, "ROSA pushers: shape overflow");
    rt->bind();
    const size_t n = steps * streams;
    uint8_t* d = io.as<uint8_t>(4 * n);
    rt->h2d(d, q, n);
    rt->h2d(d + n, k, n);
    rt->h2d(d + 2 * n, v, n);
    const push::Histories H{static_cast<push::Current*>(current.get()), static_cast<uint32_t*>(words.get()), wps};
    const uint32_t per = streams_per_warp(rt, streams);
    push_steps_kernel<<<blocks_for((streams + per - 1) / per * 32, 128), 128, 0, rt->stream>>>(H, time, steps, per, d, d + n, d + 2 * n,
                                                                                              d + 3 * n, streams);
    rt->launched("gen_push");
    rt->d2h(idx, d + 3 * n, n);
    rt->sync();
    time += steps;
}
