// One generation step - every layer, the head - as ONE kernel, a thread-block cluster per handful of sequences.
//
// A step is a chain of short stages, each bound by the latency of one f32 sum that the reference adds in order
// (LayerNorm: 2 d additions, Q / K / V, O and key: d, CMix value: dim_ffn).  As 88 kernels it took 6.5 us per kernel, two
// thirds of that launch, ramp and the first loads; as one kernel over the whole device with grid barriers a hand-over
// (barrier, then the row from L2) still cost 4 600 cycles, more than most of the sums.  Sequences are independent, so
// they need no device-wide hand-over: the CTAs of a cluster split the channels of their sequences, keep the residual rows,
// the ROSA output and the CMix hidden in shared memory, all of it in every CTA, and write their share into all of them
// (st.shared::cluster) before a cluster barrier.  Four barriers per layer:
//
//   A  LayerNorm, mixes, Q / K / V and the ROSA push of a CTA's channels
//   B  O, added to the residual rows
//   C  LayerNorm, mix, key, relu^2
//   D  value, added to the residual rows
//
// A LayerNorm is redone by every CTA (a chain costs the same once or sixteen times over).  What a stage reads from global
// memory does not depend on the step's values; it is asked for a stage ahead (weights of D into a shared-memory ring, the
// rest into L1), because one trip to L2 takes as long as 400 additions.
// All sums are the reference's, one thread per output, so the logits are those of the kernels one by one, bit for bit.
// The time-shift history is double-buffered, since every CTA reads a row of it that one of them writes anew.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

#include "common.hpp"
#include "gen_push.cuh"

namespace ullis {
namespace gen {

struct Packed {
    const uint32_t* bits;
    const uint16_t *scale, *bias;
};
struct Layer {
    const uint16_t *ln3_w, *ln3_b, *mix[3], *e, *ln2_w, *ln2_b, *ffn_mix, *value;
    Packed qkv[3], o, key;
};
struct Step {   // kernel arguments
    const Layer* layers;
    uint32_t n_layers, rows, d, ffn, vocab, time;
    uint32_t group;                                         // sequences of a cluster
    const uint32_t* tokens;                                 // page-locked host memory
    const uint16_t *embedding, *ln0_w, *ln0_b, *ln_out_w, *ln_out_b;
    Packed head;
    const float* prev_in;                                   // time-shift history [layer][2][rows][d], before and after
    float* prev_out;
    push::Histories push;
    float* logits;
};

constexpr uint32_t THREADS = 256, WARPS = THREADS / 32, MAX_GROUP = 4, MAX_CLUSTER = 16, TURN = 128;
// D: 32 outputs of a warp; a row of a piece is 16 bytes longer than its values, so that the lanes (an output each) meet no
// bank conflict
constexpr uint32_t VALUE_OUT = 32, PIECE = 128, PIECE_PITCH = PIECE * 2 + 16, PRODUCTS = 256, PRODUCT_PITCH = PRODUCTS + 4;

// Pieces of PIECE inputs in flight in D, by the bytes of one (the weights of `own` outputs); a CTA with one sum has them all.
__host__ __device__ inline uint32_t ring_stages(uint32_t group, uint32_t own, uint32_t ffn) {
    return group * own == VALUE_OUT ? ffn / PIECE : own <= 32 ? 8 : own <= 64 ? 6 : 4;
}
// Shared memory: ring | x [group][d] | y [group][d] | in [3][group][d] | act [group][ffn] | products [2][32][pitch]
inline size_t step_smem_bytes(size_t group, size_t d, size_t ffn, size_t own) {
    return ring_stages((uint32_t)group, (uint32_t)own, (uint32_t)ffn) * own * PIECE_PITCH + group * (5 * d + ffn) * 4 +
           (group * own == VALUE_OUT ? 2 * VALUE_OUT * PRODUCT_PITCH * 4 : 0);
}

__device__ __forceinline__ float h2f(uint16_t b) { return __half2float(__ushort_as_half(b)); }

__device__ __forceinline__ uint32_t cluster_size() { uint32_t n; asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n)); return n; }
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_barrier() {   // every thread of the cluster; orders the shared-memory writes
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// n floats (a multiple of 4) of each of `rows` rows, `pitch` apart, from this CTA's shared memory to the same place in
// every CTA of the cluster
__device__ __forceinline__ void share_with_cluster(const float* from, uint32_t rows, uint32_t pitch, uint32_t n) {
    const uint32_t quads = n / 4u, per_cta = rows * quads, ctas = cluster_size();
    for (uint32_t i = threadIdx.x; i < per_cta * ctas; i += THREADS) {
        const uint32_t cta = i / per_cta, q = i % per_cta;
        const float* src = from + (q / quads) * pitch + q % quads * 4u;
        const float4 v = *reinterpret_cast<const float4*>(src);
        uint32_t to;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"((uint32_t)__cvta_generic_to_shared(src)), "r"(cta));
        if (cta != cluster_rank())
            asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
    }
}
// Asks for `bytes` from p on to be in L1 by the time they are read.  (Loads whose result nobody waits for: with
// prefetch.global.L1 the later loads took as long as without.)
__device__ __forceinline__ void warm_line(uintptr_t p) {
    uint32_t unused;
    asm volatile("ld.global.ca.u32 %0, [%1];" : "=r"(unused) : "l"(p & ~(uintptr_t)3));
}
__device__ __forceinline__ void warm(const void* p, size_t bytes, uint32_t me, uint32_t threads) {
    const uintptr_t from = reinterpret_cast<uintptr_t>(p) / 128u * 128u, to = reinterpret_cast<uintptr_t>(p) + bytes;
    for (uintptr_t i = from + me * 128u; i < to; i += threads * 128u) warm_line(i < reinterpret_cast<uintptr_t>(p) ? reinterpret_cast<uintptr_t>(p) : i);
}
__device__ __forceinline__ void warm_packed(const Packed& W, uint32_t o0, uint32_t n, uint32_t K, uint32_t me, uint32_t threads) {
    warm(W.bits + ((size_t)o0 * K >> 5), (size_t)n * K / 8u, me, threads);
    warm(W.scale + o0, n * 2u, me, threads);
    if (W.bias) warm(W.bias + o0, n * 2u, me, threads);
}

// acc + v[0] + v[1] + ... + v[C - 1] in this order, by one thread; the next sixteen values are fetched while sixteen are added.
__device__ __forceinline__ float sum_in_order(const float* v, uint32_t C, float acc = 0.0f) {
    float4 a[4], b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) a[u] = *reinterpret_cast<const float4*>(v + 4 * u);
    for (uint32_t c = 0; c < C; c += 32) {   // C is a multiple of 32
#pragma unroll
        for (int u = 0; u < 4; ++u) b[u] = *reinterpret_cast<const float4*>(v + c + 16 + 4 * u);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            acc = __fadd_rn(acc, a[u].x); acc = __fadd_rn(acc, a[u].y); acc = __fadd_rn(acc, a[u].z); acc = __fadd_rn(acc, a[u].w);
        }
        const uint32_t n = c + 32 < C ? c + 32 : 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) a[u] = *reinterpret_cast<const float4*>(v + n + 4 * u);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            acc = __fadd_rn(acc, b[u].x); acc = __fadd_rn(acc, b[u].y); acc = __fadd_rn(acc, b[u].z); acc = __fadd_rn(acc, b[u].w);
        }
    }
    return acc;
}

// n rows in shared memory, normalised in place (src/model.rs:259-276); `squares` is room for as much again.  Both sums of
// a row are one thread's, in order; the squares in between are everybody's.  The warps without a row do `meanwhile` (of
// thread me of so many) under the first sum.
template <typename F>
__device__ __forceinline__ void layer_norm(float* rows, float* squares, uint32_t n, uint32_t C, const uint16_t* w, const uint16_t* b, F meanwhile) {
    __shared__ float s_mean[MAX_GROUP], s_inv[MAX_GROUP];
    const uint32_t r = threadIdx.x >> 5;
    __syncthreads();
    if (r >= n) meanwhile(threadIdx.x - n * 32u, THREADS - n * 32u);
    else if ((threadIdx.x & 31u) == 0u) s_mean[r] = __fdiv_rn(sum_in_order(rows + r * C, C), (float)C);
    __syncthreads();
    for (uint32_t k = 0; k < n; ++k) {
        const float mean = s_mean[k];
        for (uint32_t c = threadIdx.x; c < C; c += THREADS) {
            const float x = __fsub_rn(rows[k * C + c], mean);
            squares[k * C + c] = __fmul_rn(x, x);
        }
    }
    __syncthreads();
    if ((threadIdx.x & 31u) == 0u && r < n)
        s_inv[r] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(sum_in_order(squares + r * C, C), (float)C), 1e-5f)));
    __syncthreads();
    for (uint32_t c = threadIdx.x; c < C; c += THREADS) {
        const float wc = h2f(w[c]), bc = h2f(b[c]);
        for (uint32_t k = 0; k < n; ++k)
            rows[k * C + c] = __fadd_rn(__fmul_rn(__fmul_rn(__fsub_rn(rows[k * C + c], s_mean[k]), s_inv[k]), wc), bc);
    }
}

// One packed output of N rows by one thread: the sums of +/- in[i] for i ascending (src/model.rs:724-742).  The rows are
// `pitch` apart; K is a multiple of 32.
template <int N>
__device__ __forceinline__ void packed_sums(const float* in, uint32_t pitch, const uint32_t* w, uint32_t K, float (&sum)[N]) {
    constexpr int CH = 8 / N;   // 16-byte pieces of a row at a time; the next ones are on their way while these are added
    float4 x[2][N][CH];
    auto load = [&](int which, uint32_t i) {
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
            for (int u = 0; u < CH; ++u) x[which][n][u] = *reinterpret_cast<const float4*>(in + n * pitch + i + 4 * u);
    };
    uint32_t minus = ~w[0];
#pragma unroll
    for (int n = 0; n < N; ++n) sum[n] = 0.0f;
    load(0, 0);
    for (uint32_t i0 = 0; i0 < K; i0 += 64) {   // two words, so that the buffers are named at compile time
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const uint32_t i1 = i0 + 32 * half;
            if (half && i1 >= K) break;
            const uint32_t next = i1 + 32 < K ? ~w[(i1 >> 5) + 1] : 0u;
#pragma unroll
            for (int c = 0; c < N; ++c) {
                const uint32_t after = i1 + 4 * CH * (c + 1);
                load((half * N + c + 1) & 1, after < K ? after : 0u);
#pragma unroll
                for (int u = 0; u < CH; ++u) {
                    const int bit = 4 * (c * CH + u);
#pragma unroll
                    for (int n = 0; n < N; ++n) {
                        const float4 v = x[(half * N + c) & 1][n][u];
                        auto add = [&](float f, int b) {
                            sum[n] = __fadd_rn(sum[n], __uint_as_float(__float_as_uint(f) ^ (minus << (31 - b) & 0x80000000u)));
                        };
                        add(v.x, bit); add(v.y, bit + 1); add(v.z, bit + 2); add(v.w, bit + 3);
                    }
                }
            }
            minus = next;
        }
    }
}
__device__ __forceinline__ float scaled(const Packed& p, uint32_t o, float sum) {
    return __fadd_rn(p.bias ? h2f(p.bias[o]) : 0.0f, __fmul_rn(h2f(p.scale[o]), sum));
}

// LayerNorm and time-shift mixes of the cluster's rows (src/model.rs:214-228, 1331-1340, 1008-1012): in[z][n][d] from
// x[n][d]; half: 0 for the ROSA history, 1 for the CMix history.  The new history of a CTA's channels [o0, o0 + own) is its own
// to write.
template <int Z, typename F>
__device__ __forceinline__ void mixed_inputs(const Step& p, uint32_t layer, uint32_t half, uint32_t row, uint32_t n, uint32_t o0, uint32_t own,
                                             const uint16_t* ln_w, const uint16_t* ln_b, const uint16_t* const (&mix)[Z], const float* x, float* in,
                                             F meanwhile) {
    const uint32_t d = p.d;
    const size_t at = (((size_t)layer * 2 + half) * p.rows + row) * d;
    float* xs = in;   // normalised in the place of the first input, squares in that of the second (or behind the first)
    __syncthreads();
    for (uint32_t c = threadIdx.x; c < n * d; c += THREADS) xs[c] = x[c];
    layer_norm(xs, in + p.group * d, n, d, ln_w, ln_b, meanwhile);
    for (uint32_t i = threadIdx.x; i < d; i += THREADS) {   // the same thread normalised these
        float m[Z];
#pragma unroll
        for (int z = 0; z < Z; ++z) m[z] = h2f(mix[z][i]);
        for (uint32_t k = 0; k < n; ++k) {
            const uint32_t c = k * d + i;
            const float xt = xs[c], xx = p.time ? __fsub_rn(p.prev_in[at + c], xt) : -xt;
            if (i - o0 < own) p.prev_out[at + c] = xt;
#pragma unroll
            for (int z = Z - 1; z >= 0; --z) in[z * p.group * d + c] = __fadd_rn(xt, __fmul_rn(xx, m[z]));
        }
    }
    __syncthreads();
}
// `own` outputs from o0 on of a packed linear over n rows in shared memory, N rows per thread; out(row, output, value).
template <int N, typename F>
__device__ __forceinline__ void packed_outputs(const Packed& W, const float* in, uint32_t n, uint32_t K, uint32_t o0, uint32_t own, F out) {
    const uint32_t row_sets = (n + N - 1u) / N;
    for (uint32_t i = threadIdx.x; i < own * row_sets; i += THREADS) {
        const uint32_t o = o0 + i % own, r = i / own * N;
        float sum[N];
        packed_sums<N>(in + r * K, K, W.bits + ((size_t)o * K >> 5), K, sum);
#pragma unroll
        for (int k = 0; k < N; ++k)
            if (r + k < n) out(r + k, o, scaled(W, o, sum[k]));
    }
}

// Piece `piece` of the weights of the CTA's value outputs into a stage of the ring, by threads [0, threads) of which this one
// is `me`.  (One bulk copy per row of a piece was slower: 32 copies of 512 bytes took 2 400 cycles.)
__device__ __forceinline__ void fetch_value(uint8_t* stage, const uint16_t* value, uint32_t o0, uint32_t own, uint32_t ffn, uint32_t piece, uint32_t me,
                                            uint32_t threads) {
    const uint32_t to = (uint32_t)__cvta_generic_to_shared(stage);
    for (uint32_t i = me; i < own * (PIECE / 8u); i += threads) {
        const uint32_t o = i / (PIECE / 8u), g = i % (PIECE / 8u);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + o * PIECE_PITCH + g * 16u),
                     "l"(value + (size_t)(o0 + o) * ffn + piece * PIECE + g * 8u) : "memory");
    }
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

__device__ __forceinline__ float low_half(uint32_t w) { return h2f((uint16_t)(w & 0xFFFFu)); }
__device__ __forceinline__ float high_half(uint32_t w) { return h2f((uint16_t)(w >> 16)); }

// The products of PRODUCTS inputs of one row by `producers` warps (this one is number `me`), a granule of eight inputs at a
// time, lane = output; the weights are two pieces side by side.  The sums have to be added one after the other; multiplied
// they are beforehand.
__device__ __forceinline__ void value_products(const uint8_t* pieces, uint32_t piece_bytes, const float* a, uint32_t n, uint32_t me, uint32_t producers,
                                               float* products) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll 2
    for (uint32_t g = me; g < n / 8u; g += producers) {
        const uint4 w8 = *reinterpret_cast<const uint4*>(pieces + g / (PIECE / 8u) * piece_bytes + lane * PIECE_PITCH + g % (PIECE / 8u) * 16u);
        const float4 xa = *reinterpret_cast<const float4*>(a + g * 8u), xb = *reinterpret_cast<const float4*>(a + g * 8u + 4u);
        float4* to = reinterpret_cast<float4*>(products + lane * PRODUCT_PITCH + g * 8u);
        to[0] = make_float4(__fmul_rn(low_half(w8.x), xa.x), __fmul_rn(high_half(w8.x), xa.y), __fmul_rn(low_half(w8.y), xa.z), __fmul_rn(high_half(w8.y), xa.w));
        to[1] = make_float4(__fmul_rn(low_half(w8.z), xb.x), __fmul_rn(high_half(w8.z), xb.y), __fmul_rn(low_half(w8.w), xb.z), __fmul_rn(high_half(w8.w), xb.w));
    }
}
// sum + w[0] a[0] + w[1] a[1] + ... of one piece in this order, lane = output; the next granule is on its way while one is
// added.
__device__ __forceinline__ float value_piece(float sum, const uint8_t* tile, const float* a) {
    const uint4* t = reinterpret_cast<const uint4*>(tile + (threadIdx.x & 31u) * PIECE_PITCH);
    uint4 w = t[0];
    float4 xa = *reinterpret_cast<const float4*>(a), xb = *reinterpret_cast<const float4*>(a + 4);
#pragma unroll 8
    for (uint32_t g = 0; g < PIECE / 8u; ++g) {
        const uint32_t h = g + 1u < PIECE / 8u ? g + 1u : 0u;
        const uint4 w_next = t[h];
        const float4 xa_next = *reinterpret_cast<const float4*>(a + h * 8u), xb_next = *reinterpret_cast<const float4*>(a + h * 8u + 4u);
        const float p[8] = {__fmul_rn(low_half(w.x), xa.x), __fmul_rn(high_half(w.x), xa.y), __fmul_rn(low_half(w.y), xa.z), __fmul_rn(high_half(w.y), xa.w),
                            __fmul_rn(low_half(w.z), xb.x), __fmul_rn(high_half(w.z), xb.y), __fmul_rn(low_half(w.w), xb.z), __fmul_rn(high_half(w.w), xb.w)};
#pragma unroll
        for (int e = 0; e < 8; ++e) sum = __fadd_rn(sum, p[e]);
        w = w_next; xa = xa_next; xb = xb_next;
    }
    return sum;
}

// N: rows of a thread in A, C and the head
template <int N>
__global__ void __launch_bounds__(THREADS, 1)
gen_step_kernel(const Step p) {
    extern __shared__ __align__(16) uint8_t step_smem[];
    __shared__ uint8_t bits[3 * MAX_GROUP * TURN];
    __shared__ Layer layers[2];
    const uint32_t d = p.d, ffn = p.ffn, G = p.group, ctas = cluster_size(), rank = cluster_rank();
    const uint32_t own = d / ctas, o0 = rank * own;                                  // channels of this CTA
    const uint32_t f_own = ffn / ctas, f0 = rank * f_own;                            // CMix hidden units
    const uint32_t v_own = (p.vocab + ctas - 1u) / ctas, v0 = min(rank * v_own, p.vocab), v_n = min(v_own, p.vocab - v0);
    uint8_t* ring = step_smem;
    const uint32_t pieces = ffn / PIECE, tiles = own / VALUE_OUT, stages = ring_stages(G, own, ffn), stage_bytes = own * PIECE_PITCH;
    const bool alone = G * own == VALUE_OUT;   // D: one sum per CTA
    float* x = reinterpret_cast<float*>(step_smem + stages * stage_bytes);
    float* y = x + G * d;
    float* in = y + G * d;
    float* act = in + 3 * G * d;
    float* products = act + G * ffn;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    auto load_layer = [&](uint32_t l) {
        const uint32_t* from = reinterpret_cast<const uint32_t*>(p.layers + l);
        uint32_t* to = reinterpret_cast<uint32_t*>(&layers[l & 1u]);
        for (uint32_t i = threadIdx.x; i < sizeof(Layer) / 4u; i += THREADS) to[i] = from[i];
    };
    auto nothing = [](uint32_t, uint32_t) {};
    const uint32_t clusters = gridDim.x / ctas;
    for (uint32_t row = blockIdx.x / ctas * G; row < p.rows; row += clusters * G) {
        const uint32_t n = min(G, p.rows - row);
        load_layer(0);
        for (uint32_t r = 0; r < n; ++r) {   // embedding and ln0, which replaces it
            const uint16_t* e = p.embedding + (size_t)p.tokens[row + r] * d;
            for (uint32_t c = threadIdx.x; c < d; c += THREADS) x[r * d + c] = h2f(e[c]);
        }
        layer_norm(x, in, n, d, p.ln0_w, p.ln0_b, nothing);
        // the pushes of a turn of at most 128 channels: `per` channels side by side of one row for a warp at a time
        const uint32_t turn = min(TURN, own);
        uint32_t per = 1u;
        while (per < 32u && 2u * per <= n * turn / WARPS) per *= 2u;   // turn is a multiple of 32
        auto push_set = [&](uint32_t l, uint32_t c0, uint32_t j, size_t& stream, uint32_t& r, uint32_t& c) {
            r = j / (turn / per);
            c = j % (turn / per) * per + lane;
            stream = ((size_t)l * p.rows + row + r) * d + o0 + c0 + c - lane;
            return lane < per && r < n && c0 + c < own;
        };
        auto push_begin = [&](uint32_t l) {   // of this warp's first set: asked for while something else is waited for
            size_t stream;
            uint32_t r, c;
            const bool live = push_set(l, 0u, warp, stream, r, c);
            return push::begin(p.push, stream, live, p.time);
        };
        push::Ahead ahead = push_begin(0u);
        for (uint32_t l = 0; l < p.n_layers; ++l) {
            __syncthreads();   // the layer's pointers; the ring is free
            const Layer& L = layers[l & 1u];
            // ---- A
            mixed_inputs<3>(p, l, 0u, row, n, o0, own, L.ln3_w, L.ln3_b, L.mix, x, in, [&](uint32_t me, uint32_t threads) {
                // what A, B and C read from global memory
                const size_t at = ((size_t)l * 2 * p.rows + row) * d;
                auto all = [&](const void* from, size_t bytes) { warm(from, bytes, me, threads); };
                all(L.ln3_w, d * 2u); all(L.ln3_b, d * 2u);
                if (p.time) all(p.prev_in + at, (size_t)n * d * 4u);
                for (int z = 0; z < 3; ++z) {
                    all(L.mix[z], d * 2u);
                    warm_packed(L.qkv[z], o0, own, d, me, threads);
                }
                all(L.e + o0, own * 2u);
                for (uint32_t i = me; i < n * own; i += threads)   // the keys of this CTA's streams, for a search
                    warm(p.push.of(((size_t)l * p.rows + row + i / own) * d + o0 + i % own, 1), (p.time / 32u + 1u) * 4u, 0u, 1u);
                warm_packed(L.o, o0, own, d, me, threads);
                all(L.ln2_w, d * 2u); all(L.ln2_b, d * 2u); all(L.ffn_mix, d * 2u);
                if (p.time) all(p.prev_in + at + (size_t)p.rows * d, (size_t)n * d * 4u);
                warm_packed(L.key, f0, f_own, d, me, threads);
            });
            for (uint32_t c0 = 0; c0 < own; c0 += turn) {
                const uint32_t nc = min(turn, own - c0), row_sets = (n + N - 1u) / N;
                for (uint32_t i = threadIdx.x; i < 3u * nc * row_sets; i += THREADS) {
                    const uint32_t z = i / nc % 3u, c = i % nc, r = i / (3u * nc) * N, o = o0 + c0 + c;
                    const Packed& W = L.qkv[z];
                    float sum[N];
                    packed_sums<N>(in + (z * G + r) * d, d, W.bits + ((size_t)o * d >> 5), d, sum);
#pragma unroll
                    for (int k = 0; k < N; ++k)
                        if (r + k < n) bits[(z * MAX_GROUP + r + k) * TURN + c] = scaled(W, o, sum[k]) > 0.0f;   // src/rosa.rs:372-374
                }
                __syncthreads();
                for (uint32_t j = warp; j < n * (turn / per); j += WARPS) {
                    size_t stream;
                    uint32_t r, c;
                    const bool live = push_set(l, c0, j, stream, r, c);
                    if (j != warp || c0) ahead = push::begin(p.push, stream, live, p.time);
                    const uint32_t at = r * TURN + c;
                    const bool idx = push::step(p.push, stream, live, p.time, ahead, live ? bits[at] : 0u, live ? bits[MAX_GROUP * TURN + at] : 0u,
                                                live ? bits[2 * MAX_GROUP * TURN + at] : 0u);
                    if (live) {   // src/model.rs:1344-1351
                        const float ev = h2f(L.e[o0 + c0 + c]);
                        y[r * d + o0 + c0 + c] = idx ? ev : -ev;
                    }
                }
                __syncthreads();
            }
            share_with_cluster(y + o0, n, d, own);
            cluster_barrier();
            // ---- B
            // The first pieces of D's weights, by the threads that have no output here if there are enough of them.  (A thread
            // waits for its own copies; one that took no part has none to wait for.)
            const uint32_t busy = min((n * own + 31u) / 32u * 32u, THREADS / 2u), first = alone ? pieces : stages - 1u;
            if (threadIdx.x >= busy)
                for (uint32_t k = 0; k < first; ++k) {
                    if (k < pieces) fetch_value(ring + k * stage_bytes, L.value, o0, own, ffn, k, threadIdx.x - busy, THREADS - busy);
                    copies_commit();
                }
            packed_outputs<1>(L.o, y, n, d, o0, own, [&](uint32_t r, uint32_t o, float v) { x[r * d + o] = __fadd_rn(x[r * d + o], v); });
            __syncthreads();
            share_with_cluster(x + o0, n, d, own);
            cluster_barrier();
            // ---- C
            const uint16_t* const ffn_mix[1] = {L.ffn_mix};
            mixed_inputs<1>(p, l, 1u, row, n, o0, own, L.ln2_w, L.ln2_b, ffn_mix, x, in, nothing);
            packed_outputs<N>(L.key, in, n, d, f0, f_own, [&](uint32_t r, uint32_t o, float v) {
                const float m = fmaxf(v, 0.0f);   // src/model.rs:999
                act[r * ffn + o] = __fmul_rn(m, m);
            });
            __syncthreads();
            share_with_cluster(act + f0, n, ffn, f_own);
            if (l + 1u < p.n_layers) load_layer(l + 1u);
            cluster_barrier();
            // ---- D
            if (alone) {
                // One warp adds, the others multiply for it, PRODUCTS inputs ahead: it is then as fast as its chain of additions.
                asm volatile("cp.async.wait_all;" ::: "memory");
                float sum = 0.0f;
                for (uint32_t k = 0; k < ffn + PRODUCTS; k += PRODUCTS) {
                    float* of = products + (k / PRODUCTS & 1u) * VALUE_OUT * PRODUCT_PITCH;
                    const float* before = products + (~(k / PRODUCTS) & 1u) * VALUE_OUT * PRODUCT_PITCH;
                    __syncthreads();
                    if (warp != 0u) {
                        if (k < ffn) value_products(ring + k / PIECE * stage_bytes, stage_bytes, act + k, min(PRODUCTS, ffn - k), warp - 1u, WARPS - 1u, of);
                    } else if (k) {
                        sum = sum_in_order(before + lane * PRODUCT_PITCH, min(PRODUCTS, ffn - (k - PRODUCTS)), sum);   // src/model.rs:419-436
                    }
                }
                if (warp == 0u) x[o0 + lane] = __fadd_rn(x[o0 + lane], sum);
            }
            // A warp adds up 32 outputs of a row.
            const uint32_t sums = n * tiles;
            for (uint32_t k0 = 0; k0 < sums && !alone; k0 += WARPS) {
                if (k0) {   // more sums than warps: the weights once more
                    __syncthreads();
                    for (uint32_t k = 0; k < stages - 1u; ++k) {
                        if (k < pieces) fetch_value(ring + k * stage_bytes, L.value, o0, own, ffn, k, threadIdx.x, THREADS);
                        copies_commit();
                    }
                }
                const uint32_t mine = k0 + warp, tile = mine % tiles, r = mine / tiles;
                float sum = 0.0f;
                uint32_t at = 0;   // piece k lies in stage k % stages
                for (uint32_t k = 0; k < pieces; ++k) {
                    // one group is committed per piece, so all but the newest stages - 2 having landed means piece k has
                    if (stages == 8u) asm volatile("cp.async.wait_group 6;" ::: "memory");
                    else if (stages == 6u) asm volatile("cp.async.wait_group 4;" ::: "memory");
                    else asm volatile("cp.async.wait_group 2;" ::: "memory");
                    __syncthreads();   // piece k is everybody's; piece k - 1 is done with
                    if (k + stages - 1u < pieces)
                        fetch_value(ring + (at ? at - 1u : stages - 1u) * stage_bytes, L.value, o0, own, ffn, k + stages - 1u, threadIdx.x, THREADS);
                    copies_commit();
                    if (mine < sums) sum = value_piece(sum, ring + at * stage_bytes + tile * VALUE_OUT * PIECE_PITCH, act + r * ffn + k * PIECE);
                    at = at + 1u < stages ? at + 1u : 0u;
                }
                if (mine < sums) {
                    float* to = x + r * d + o0 + tile * VALUE_OUT + lane;
                    *to = __fadd_rn(*to, sum);
                }
            }
            __syncthreads();
            share_with_cluster(x + o0, n, d, own);
            if (l + 1u < p.n_layers) ahead = push_begin(l + 1u);
            cluster_barrier();
        }
        layer_norm(x, in, n, d, p.ln_out_w, p.ln_out_b, [&](uint32_t me, uint32_t threads) { warm_packed(p.head, v0, v_n, d, me, threads); });
        __syncthreads();
        packed_outputs<N>(p.head, x, n, d, v0, v_n, [&](uint32_t r, uint32_t o, float v) { p.logits[(size_t)(row + r) * p.vocab + o] = v; });
        cluster_barrier();   // the rows are written anew only when nobody reads them
    }
}

}  // namespace gen
}  // namespace ullis
