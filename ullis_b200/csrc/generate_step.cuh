// One generation step - every layer, the head - as ONE kernel, a thread-block cluster per handful of sequences.
//
// A step is a chain of short stages, each bound by f32 sums that the reference adds in order (LayerNorm: 2 d additions,
// Q / K / V, O and key: d, CMix value: dim_ffn).  As 88 kernels it took 6.5 us per kernel, two thirds of that launch, ramp
// and the first loads; as one kernel over the whole device with grid barriers a hand-over (barrier, then the row from L2)
// still cost 4 600 cycles, more than most of the sums.  Sequences are independent, so they need no device-wide hand-over:
// the CTAs of a cluster split the channels of their sequences, keep the residual rows, the ROSA output and the CMix hidden
// in shared memory, all of it in every CTA, and send their share to all of them (st.async, counted on a barrier of the receiver).
// Four of these exchanges per layer:
//
//   A  LayerNorm, mixes, Q / K / V and the ROSA push of a CTA's channels
//   B  O, added to the residual rows
//   C  LayerNorm, mix, key, relu^2
//   D  value, added to the residual rows
//
// A CTA that has received a stage's shares knows that every other one is done with the stage before, so an exchange orders the
// reads of a buffer before its next writes as a cluster barrier would (in 700 cycles instead of 1 600).
// A LayerNorm is redone by every CTA (a chain costs the same once or sixteen times over).  What a stage reads from global
// memory does not depend on the step's values: the weights are copied to shared memory a stage ahead by the copy engine (with
// cp.async the issuing threads stood still for 4 500 cycles per layer), and LayerNorm's vectors and the time-shift history go
// to registers before its sums.
//
// With one row per thread and output a sum takes 4.4 to 5 cycles per term, the latency of the addition; with more rows and
// outputs in a cluster it is issue slots and shared-memory reads that count.  Therefore the rows of a cluster lie side by side
// per channel, a thread adds up all of them for J outputs at once, and two rows take one fma.f32x2 (512 inputs, 1024 sums of
// a CTA: one output and two scalar rows per thread 22 000 cycles, four outputs and a pair of rows 11 000).
// All layers run the same code, and what of it does not fit the instruction cache of an SM is fetched again in every one (with
// a copy of the sums per stage, 160 KB in all, 1 000 misses per layer).  So A, B and C are three turns of one loop, and loops are
// unrolled only as far as a sum needs it; a function that is not inlined costs more (550 cycles per call).
// All sums are the reference's, so the logits are those of the kernels one by one, bit for bit: x * +-1 is exact, so
// fma(x, +-1, sum) rounds what sum +- x does.
// The time-shift history is double-buffered, since every CTA reads a row of it that one of them writes anew.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

#include <type_traits>

#include "common.hpp"
#include "gen_push.cuh"
#include "tc_ptx.cuh"

namespace ullis {
namespace gen {

struct Packed {
    const uint32_t* bits;
    const uint16_t *scale, *bias;
};
struct Layer {
    const uint16_t *ln3_w, *ln3_b, *mix[3], *e, *ln2_w, *ln2_b, *ffn_mix;
    Packed qkv[3], o, key;
};
struct Step {   // kernel arguments
    const Layer* layers;
    const CUtensorMap* values;                              // of the layers' value matrices by slabs (tc::slab_map)
    uint32_t n_layers, rows, d, ffn, vocab, time;
    uint32_t stages;                                        // of the ring of D
    uint32_t staged;                                        // packed weights go through shared memory
    uint32_t polls;                                         // of a wait, before it gives up
    float minus_zero;                                       // -0.0f, unknown to the compiler (value_piece)
    const uint32_t* tokens;                                 // page-locked host memory
    const uint16_t *embedding, *ln0_w, *ln0_b, *ln_out_w, *ln_out_b;
    Packed head;
    const float* prev_in;                                   // time-shift history [layer][2][rows][d], before and after
    float* prev_out;
    push::Histories push;
    float* logits;
    uint32_t* status;                                       // page-locked host memory
};

constexpr uint32_t THREADS = 256, WARPS = THREADS / 32, MAX_GROUP = 4, MAX_CLUSTER = 16;
// D: 32 outputs of a warp.  Weights come in pieces of 128 inputs of all of a CTA's outputs: slab by slab of 64 inputs, output by
// output, and 16-byte granule g of output o lies at g ^ (o % 8) (the copy engine's 128-byte swizzle: the lanes, an output each,
// meet no bank conflict).  A piece is one copy, since each of them holds the asking warp, and the shared memory it works on, up.  A CTA with 32 sums in all has one warp add what the others have multiplied, PRODUCTS inputs at a time.
constexpr uint32_t VALUE_OUT = 32, PIECE = 128, SLAB = 64, BOX_BYTES = SLAB * VALUE_OUT * 2, PRODUCTS = PIECE, PRODUCT_PITCH = PRODUCTS + 4, PRODUCT_SLOTS = 3;
constexpr uint32_t VALUE_BODY = 8;   // granules of the loop body of D
constexpr uint32_t MAX_STAGES = 32;

__host__ __device__ inline uint32_t most(uint32_t a, uint32_t b) { return a > b ? a : b; }
// Floats of a row: the residual row, the first input (where the squares of LayerNorm lie before it), and one region for the
// CMix hidden (C, D), the ROSA output (A, B) and the other two inputs (A).
__host__ __device__ inline uint32_t row_floats(uint32_t d, uint32_t ffn) { return 2u * d + most(ffn, 3u * d); }

// How a CTA's shared memory is laid out: ring | products | rows | bits of q, k and v | Q/K/V or key weights | O weights.
struct Layout {
    uint32_t ring, products, rows, bits, wide, o, total;   // byte offsets
    __host__ __device__ Layout(uint32_t group, uint32_t d, uint32_t ffn, uint32_t ctas, uint32_t stages, bool staged) {
        const uint32_t own = d / ctas;
        ring = 0;
        products = ring + stages * own * (PIECE * 2u);
        rows = products + (group * own == VALUE_OUT ? PRODUCT_SLOTS * VALUE_OUT * PRODUCT_PITCH * 4u : 0u);
        bits = rows + group * row_floats(d, ffn) * 4u;
        wide = bits + 3u * group * own;
        o = wide + (staged ? most(3u * own, ffn / ctas) * (d / 8u) : 0u);
        total = o + (staged ? own * (d / 8u) : 0u) + 1024u;   // the ring starts on a border of 1024 bytes
    }
};
// Pieces of D's weights in flight: as many as fit, up to 8; a CTA with one sum per lane of a warp has them all.
inline uint32_t ring_stages(uint32_t group, uint32_t d, uint32_t ffn, uint32_t ctas, bool staged, size_t limit) {
    if (group * d / ctas == VALUE_OUT) return ffn / PIECE;
    for (uint32_t s : {8u, 6u, 4u, 3u})
        if (Layout(group, d, ffn, ctas, s, staged).total <= limit) return s;
    return 2u;
}

__device__ __forceinline__ float h2f(uint16_t b) { return __half2float(__ushort_as_half(b)); }

__device__ __forceinline__ uint32_t cluster_size() { uint32_t n; asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n)); return n; }
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
// Every thread of the cluster.
__device__ __forceinline__ void cluster_arrive() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The copies of a CTA, issued by one thread, and the waits for them.  gave_up: where a wait of this CTA, or of another one of its
// cluster, ran out.  Nobody waits, asks for copies or sends any more then: an mbarrier whose phase is not over must not be told to
// expect the next one.  The stages run to their end on what lies in shared memory, which decides no address and no loop, so that
// everybody passes the same barriers; the step reports the failure.
constexpr uint32_t BARS = 2 * MAX_STAGES + 7, MAX_BOX = 256;
struct Copies {
    uint64_t ring[BARS];   // mbarriers: a stage of the ring is full, is empty, one for each set of packed weights, for each exchange
    __device__ uint64_t* empty() { return ring + MAX_STAGES; }
    __device__ uint64_t* qkv_o() { return ring + 2 * MAX_STAGES; }
    __device__ uint64_t* key() { return ring + 2 * MAX_STAGES + 1; }
    __device__ uint64_t* head() { return ring + 2 * MAX_STAGES + 2; }
    __device__ uint64_t* exchange(uint32_t stage) { return ring + 2 * MAX_STAGES + 3 + stage; }   // after A, B, C, D
    uint32_t gave_up;
};
__device__ __forceinline__ bool has_given_up(const Copies& copies) { return *static_cast<const volatile uint32_t*>(&copies.gave_up) != 0u; }
__device__ __forceinline__ void copies_wait(Copies& copies, uint64_t* bar, uint32_t phase, const Step& p, uint32_t site) {
    uint32_t polls = 0;
#pragma unroll 1
    do {
        if (polls < p.polls && ptx::mbar_try_wait(bar, phase & 1u)) return;
        if (has_given_up(copies)) return;
    } while (polls++ < p.polls);
    *static_cast<volatile uint32_t*>(&copies.gave_up) = site;
}
// n floats (a multiple of 4) of each of `rows` rows, `pitch` apart, from this CTA's shared memory to the same place in every
// other CTA of the cluster, a CTA per warp at a time, counted on the receiver's barrier `bar`.  One thread says what this CTA's own
// barrier has to wait for.  false: nothing was sent, after a give-up.
__device__ __forceinline__ bool send_to_cluster(const float* from, uint32_t rows, uint32_t pitch, uint32_t n, Copies& copies, uint64_t* bar) {
    const uint32_t ctas = cluster_size(), me = cluster_rank(), lane = threadIdx.x & 31u;
    if (has_given_up(copies)) return false;
    if (threadIdx.x == 0u) ptx::mbar_arrive_expect_tx(bar, (ctas - 1u) * rows * n * 4u);
#pragma unroll 1
    for (uint32_t cta = threadIdx.x >> 5; cta < ctas; cta += WARPS) {
        if (cta == me) continue;
        const uint32_t to = ptx::cluster_map(from, cta), counted = ptx::cluster_map(bar, cta);
#pragma unroll 1
        for (uint32_t r = 0; r < rows; ++r)
#pragma unroll 1
            for (uint32_t q = 4u * lane; q < n; q += 128u) {
                const float4 v = *reinterpret_cast<const float4*>(from + r * pitch + q);
                asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(to + (r * pitch + q) * 4u),
                             "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(counted) : "memory");
            }
    }
    return true;
}
// `bytes` (a multiple of 16, like both addresses) to shared memory by the copy engine, counted on `bar`.
__device__ __forceinline__ void copy_bytes(void* to, const void* from, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(ptx::smem_u32(to)), "l"(from), "r"(bytes),
                 "r"(ptx::smem_u32(bar)) : "memory");
}
// Asks for `bytes` from p on to be in L1 by the time they are read.  (Loads whose result nobody waits for: with
// prefetch.global.L1 the later loads took as long as without.)
__device__ __forceinline__ void warm_line(uintptr_t p) {
    uint32_t unused;
    asm volatile("ld.global.ca.u32 %0, [%1];" : "=r"(unused) : "l"(p & ~(uintptr_t)3));
}
__device__ __forceinline__ void warm(const void* p, uint32_t bytes) {
    const uintptr_t to = reinterpret_cast<uintptr_t>(p) + bytes;
#pragma unroll 1
    for (uintptr_t i = reinterpret_cast<uintptr_t>(p); i < to; i = i / 128u * 128u + 128u) warm_line(i);
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

// Mean and 1 / sqrt(variance + eps) of a row (src/model.rs:259-276) by a warp, in its first lane: both sums in order by one lane,
// the squares in between by all of them, into `squares`.
__device__ __forceinline__ float2 row_statistics(const float* row, float* squares, uint32_t C) {
    const uint32_t lane = threadIdx.x & 31u;
    float mean = 0.0f;
#pragma unroll 1
    for (int pass = 0;; ++pass) {
        float average = 0.0f;
        if (lane == 0u) average = __fdiv_rn(sum_in_order(pass ? squares : row, C), (float)C);
        if (pass) return make_float2(mean, __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(average, 1e-5f))));
        mean = __shfl_sync(0xFFFFFFFFu, average, 0);
#pragma unroll 1
        for (uint32_t c = 4u * lane; c < C; c += 128u) {
            float4 x = *reinterpret_cast<const float4*>(row + c);
            x.x = __fsub_rn(x.x, mean); x.y = __fsub_rn(x.y, mean); x.z = __fsub_rn(x.z, mean); x.w = __fsub_rn(x.w, mean);
            *reinterpret_cast<float4*>(squares + c) = make_float4(__fmul_rn(x.x, x.x), __fmul_rn(x.y, x.y), __fmul_rn(x.z, x.z), __fmul_rn(x.w, x.w));
        }
        __syncwarp();
    }
}
__device__ __forceinline__ float normalised(float x, float mean, float inv, float w, float b) {
    return __fadd_rn(__fmul_rn(__fmul_rn(__fsub_rn(x, mean), inv), w), b);
}

__device__ __forceinline__ uint32_t load_ahead(const void* p) {   // issued here, not where the value is needed
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t load_half_ahead(const uint16_t* p) {
    uint32_t v;
    asm volatile("ld.global.u16 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float low_half(uint32_t w) { return h2f((uint16_t)(w & 0xFFFFu)); }
__device__ __forceinline__ float high_half(uint32_t w) { return h2f((uint16_t)(w >> 16)); }

// The statistics of the rows x[r * d] by a warp each; true for the threads that have none to do.
struct Statistics {
    float mean[MAX_GROUP], inv[MAX_GROUP];
};
__device__ __forceinline__ bool rows_statistics(const float* x, float* squares, uint32_t n, uint32_t d, Statistics& s) {
    const uint32_t r = threadIdx.x >> 5;
    if (r >= n) return true;
    const float2 v = row_statistics(x + r * d, squares + r * d, d);
    if ((threadIdx.x & 31u) == 0u) { s.mean[r] = v.x; s.inv[r] = v.y; }
    return false;
}

// LayerNorm and time-shift mixes of the cluster's rows (src/model.rs:214-228, 1331-1340, 1008-1012): input z of row r and channel c
// to in[z * apart + c * G + r] from x[r * d + c].  half: 0 for ROSA (three inputs, its history), 1 for the CMix (one).  The new
// history of a CTA's channels [o0, o0 + own) is its own to write.  A thread has two channels side by side at a time; what it reads
// from global memory for the first ones is asked for before the sums.
template <int G>
__device__ __forceinline__ void mixed_inputs(const Step& p, const Layer& L, uint32_t layer, uint32_t half, uint32_t row, uint32_t n, uint32_t o0, uint32_t own,
                                          const float* x, float* in, uint32_t apart) {
    __shared__ Statistics stats;
    const uint32_t d = p.d, inputs = half ? 1u : 3u;
    const size_t at = (((size_t)layer * 2 + half) * p.rows + row) * d;
    const uint16_t *ln_w = half ? L.ln2_w : L.ln3_w, *ln_b = half ? L.ln2_b : L.ln3_b, *mix0 = half ? L.ffn_mix : L.mix[0];
    uint32_t w, b, m[3];
    float2 before[G];
    auto ask = [&](uint32_t c) {
        w = load_ahead(ln_w + c);
        b = load_ahead(ln_b + c);
        m[0] = load_ahead(mix0 + c);
        if (inputs > 1u) {
            m[1] = load_ahead(L.mix[1] + c);
            m[2] = load_ahead(L.mix[2] + c);
        }
#pragma unroll
        for (int r = 0; r < G; ++r)
            if (p.time && r < n)
                asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(before[r].x), "=f"(before[r].y) : "l"(p.prev_in + at + (size_t)r * d + c));
    };
    uint32_t c = 2u * threadIdx.x;
    if (c < d) ask(c);
    __syncthreads();
    if (rows_statistics(x, in, n, d, stats) && !half) {
        // the keys of this CTA's streams, for a search, and the v bits it leads to
        const uint32_t threads = THREADS - n * 32u;
#pragma unroll 1
        for (uint32_t i = threadIdx.x - n * 32u; i < n * own; i += threads) {
            const size_t stream = ((size_t)layer * p.rows + row + i / own) * d + o0 + i % own;
            warm(p.push.of(stream, 1), (p.time / 32u + 1u) * 4u);
            warm(p.push.of(stream, 2), (p.time / 32u + 1u) * 4u);
        }
    }
    __syncthreads();
#pragma unroll 1
    while (c < d) {
#pragma unroll
        for (int r = 0; r < G; ++r) {
            if (r >= n) break;
            const float2 v = *reinterpret_cast<const float2*>(x + r * d + c);
            const float a = normalised(v.x, stats.mean[r], stats.inv[r], low_half(w), low_half(b));
            const float e = normalised(v.y, stats.mean[r], stats.inv[r], high_half(w), high_half(b));
            const float da = p.time ? __fsub_rn(before[r].x, a) : -a, de = p.time ? __fsub_rn(before[r].y, e) : -e;
            if (c - o0 < own) *reinterpret_cast<float2*>(p.prev_out + at + (size_t)r * d + c) = make_float2(a, e);
#pragma unroll
            for (int z = 0; z < 3; ++z) {
                if (z >= inputs) break;
                in[z * apart + c * G + r] = __fadd_rn(a, __fmul_rn(da, low_half(m[z])));
                in[z * apart + (c + 1u) * G + r] = __fadd_rn(e, __fmul_rn(de, high_half(m[z])));
            }
        }
        c += 2u * THREADS;
        if (c < d) ask(c);
    }
}

__device__ __forceinline__ float2 fma_pair(float2 a, float2 b, float2 c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)), "l"(*reinterpret_cast<uint64_t*>(&c)));
    return *reinterpret_cast<float2*>(&r);
}
__device__ __forceinline__ float2 add_pair(float2 a, float2 b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)));
    return *reinterpret_cast<float2*>(&r);
}
// The sign of x turned unless the top bit of `bits` is set, and 1.0 with that sign, as one instruction each.
__device__ __forceinline__ uint32_t flip_unless(uint32_t bits, uint32_t x) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xA6;" : "=r"(r) : "r"(bits), "r"(0x80000000u), "r"(x));   // (~a & b) ^ c
    return r;
}
__device__ __forceinline__ uint32_t minus_unless(uint32_t bits) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xAE;" : "=r"(r) : "r"(bits), "r"(0x80000000u), "r"(0x3F800000u));   // (~a & b) | c
    return r;
}
__device__ __forceinline__ float& lane_of(float4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// Four words of a packed row, of which `left` are there.
__device__ __forceinline__ uint4 four_words(const uint32_t* w, uint32_t left, bool quads) {
    if (quads) return *reinterpret_cast<const uint4*>(w);
    return make_uint4(w[0], left > 1u ? w[1] : 0u, left > 2u ? w[2] : 0u, left > 3u ? w[3] : 0u);
}
// The sums of +/- in[i] for i ascending (src/model.rs:724-742) of G rows side by side (input i of row r at i * G + r) for J
// outputs; output j takes its inputs from in + j * apart and their signs from w + j * w_apart, in shared or global memory.  K is a
// multiple of 32.  The inputs of the next CH terms and the next four words are on their way while these are added.
template <int G, int J, bool APART>
__device__ __forceinline__ void packed_sums(const float* in, uint32_t apart, const uint32_t* w, uint32_t w_apart, uint32_t K, float (&sum)[J][G]) {
    constexpr int S = APART ? J : 1, BODY = G * J == 1 ? 64 : 32, CH = G * J == 1 ? 16 : G == 1 ? 8 : (G * S > 4 || J * G > 8) ? 4 : 8, Q = CH * G / 4;
    const uint32_t words = K / 32u;
    const bool quads = words % 4u == 0u;
    float4 x[2][S][Q];
    float total[J][G];
    uint4 now[J], next[J];
    auto load = [&](int which, uint32_t i) {
#pragma unroll
        for (int s = 0; s < S; ++s)
#pragma unroll
            for (int q = 0; q < Q; ++q) x[which][s][q] = *reinterpret_cast<const float4*>(in + s * apart + i * G + 4 * q);
    };
#pragma unroll
    for (int j = 0; j < J; ++j) {
        next[j] = four_words(w + j * w_apart, words, quads);
#pragma unroll
        for (int r = 0; r < G; ++r) total[j][r] = 0.0f;
    }
    load(0, 0u);
#pragma unroll 1
    for (uint32_t i = 0; i < K; i += BODY) {
        if (i % 128u == 0u) {
            const uint32_t then = i + 128u < K ? i / 32u + 4u : 0u;
#pragma unroll
            for (int j = 0; j < J; ++j) {
                now[j] = next[j];
                next[j] = four_words(w + j * w_apart + then, words - then, quads);
            }
        }
#pragma unroll
        for (int c = 0; c < BODY / CH; ++c) {
            if (BODY == 64 && c == 32 / CH && i + 32u >= K) break;   // K an odd number of words
            const uint32_t after = i + CH * (c + 1);
            load((c & 1) ^ 1, after < K ? after : 0u);
#pragma unroll
            for (int e = 0; e < CH; ++e)
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    const uint32_t up = (c * CH + e < 32 ? now[j].x : now[j].y) << (31 - (c * CH + e) % 32);   // the sign on top: 1 is +
                    if (G == 1) {
                        const float v = lane_of(x[c & 1][APART ? j : 0][e / 4], e % 4);
                        total[j][0] = __fadd_rn(total[j][0], __uint_as_float(flip_unless(up, __float_as_uint(v))));
                    } else {
                        const float sign = __uint_as_float(minus_unless(up));
#pragma unroll
                        for (int r = 0; r < G; r += 2) {
                            const int q = e * G + r, r1 = r + 1 < G ? r + 1 : 0;
                            const float2 v = make_float2(lane_of(x[c & 1][APART ? j : 0][q / 4], q % 4), lane_of(x[c & 1][APART ? j : 0][q / 4], (q + 1) % 4));
                            const float2 s = fma_pair(v, make_float2(sign, sign), make_float2(total[j][r], total[j][r1]));
                            total[j][r] = s.x;
                            total[j][r1] = s.y;
                        }
                    }
                }
        }
#pragma unroll
        for (int j = 0; j < J; ++j) {
            if (BODY == 32) {
                now[j].x = now[j].y; now[j].y = now[j].z; now[j].z = now[j].w;
            } else {
                now[j].x = now[j].z; now[j].y = now[j].w;
            }
        }
    }
#pragma unroll
    for (int j = 0; j < J; ++j)
#pragma unroll
        for (int r = 0; r < G; ++r) sum[j][r] = total[j][r];
}

// n_out outputs of a packed linear over G rows, J per thread (n_out a multiple of J); `first`: where they begin in scale and bias;
// emit(output, row, value) with the output counted from 0.
template <int G, int J, typename F>
__device__ __forceinline__ void packed_outputs(const Packed& P, const uint32_t* w, const float* in, uint32_t n, uint32_t K, uint32_t first, uint32_t n_out,
                                               F emit) {
    const uint32_t apart = n_out / J;
#pragma unroll 1
    for (uint32_t o = threadIdx.x; o < apart; o += THREADS) {
        uint32_t scale[J], bias[J];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            scale[j] = load_half_ahead(P.scale + first + o + j * apart);
            bias[j] = P.bias ? load_half_ahead(P.bias + first + o + j * apart) : 0u;
        }
        float sum[J][G];
        packed_sums<G, J, false>(in, 0u, w + (size_t)o * (K / 32u), apart * (K / 32u), K, sum);
#pragma unroll
        for (int j = 0; j < J; ++j)
#pragma unroll
            for (int r = 0; r < G; ++r)
                if (r < n) emit(o + j * apart, (uint32_t)r, __fadd_rn(low_half(bias[j]), __fmul_rn(low_half(scale[j]), sum[j][r])));
    }
}

// `slabs` slabs (as many as the map's box has) from slab `slab` on of the weights of the value outputs [o0, o0 + own), by one thread.
__device__ __forceinline__ void fetch_value(uint8_t* to, const CUtensorMap* map, uint32_t o0, uint32_t own, uint32_t slab, uint32_t slabs, uint64_t* bar) {
    ptx::mbar_arrive_expect_tx(bar, slabs * own * (SLAB * 2u));
    const uint32_t rows = min(own, MAX_BOX);
    if (rows == own) {
        ptx::tma_load_3d(to, map, bar, 0, (int32_t)o0, (int32_t)slab);
    } else {   // the box is one slab of MAX_BOX outputs
#pragma unroll 1
        for (uint32_t b = 0; b < slabs * (own / rows); ++b)
            ptx::tma_load_3d(to + b * rows * (SLAB * 2u), map, bar, 0, (int32_t)(o0 + b % (own / rows) * rows), (int32_t)(slab + b / (own / rows)));
    }
}
// Where the lane's output of a tile has its granules in the box of a slab (shared address): granule g (eight inputs) at
// granules ^ 16 g.
__device__ __forceinline__ uint32_t lane_granules(const uint8_t* box) {
    const uint32_t lane = threadIdx.x & 31u;
    return ptx::smem_u32(box) + lane * 128u + (lane & 7u) * 16u;
}
__device__ __forceinline__ uint4 granule(uint32_t granules, uint32_t g) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(granules ^ 16u * g));
    return v;
}

__device__ __forceinline__ void barrier_arrive(uint32_t id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(THREADS) : "memory"); }
__device__ __forceinline__ void barrier_sync(uint32_t id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(THREADS) : "memory"); }

// The products of PRODUCTS inputs of one row by `producers` warps (this one is number `me`), a granule of eight inputs at a
// time, lane = output.  The sums have to be added one after the other; multiplied they are beforehand.
__device__ __forceinline__ void value_products(const uint8_t* piece, const float* a, uint32_t me, uint32_t producers, float* products) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll 3
    for (uint32_t g = me; g < PRODUCTS / 8u; g += producers) {
        const uint4 w8 = granule(lane_granules(piece + g / 8u * BOX_BYTES), g % 8u);
        const float4 xa = *reinterpret_cast<const float4*>(a + g * 8u), xb = *reinterpret_cast<const float4*>(a + g * 8u + 4u);
        float4* to = reinterpret_cast<float4*>(products + lane * PRODUCT_PITCH + g * 8u);
        to[0] = make_float4(__fmul_rn(low_half(w8.x), xa.x), __fmul_rn(high_half(w8.x), xa.y), __fmul_rn(low_half(w8.y), xa.z), __fmul_rn(high_half(w8.y), xa.w));
        to[1] = make_float4(__fmul_rn(low_half(w8.z), xb.x), __fmul_rn(high_half(w8.z), xb.y), __fmul_rn(low_half(w8.w), xb.z), __fmul_rn(high_half(w8.w), xb.w));
    }
}
// The 32 sums of a CTA that has no more (src/model.rs:419-436): warp 0 adds, the others multiply for it into PRODUCT_SLOTS
// slots, handed over by named barriers (1 + slot: full, 4 + slot: empty).  Returns the sum of the lane's output in warp 0.
__device__ __forceinline__ float value_alone(const uint8_t* ring, Copies& copies, uint32_t phase, const float* act, uint32_t pieces, float* products, const Step& p) {
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    constexpr uint32_t FULL = 1u, EMPTY = FULL + PRODUCT_SLOTS, SLOT = VALUE_OUT * PRODUCT_PITCH;
    float sum = 0.0f;
    uint32_t slot = 0;
    copies_wait(copies, copies.ring, phase, p, 0x601u);
    if (warp != 0u) {
#pragma unroll 1
        for (uint32_t k = 0; k < pieces; ++k) {
            if (k >= PRODUCT_SLOTS) barrier_sync(EMPTY + slot);
            value_products(ring + k * (VALUE_OUT * PIECE * 2u), act + k * PIECE, warp - 1u, WARPS - 1u, products + slot * SLOT);
            barrier_arrive(FULL + slot);
            slot = slot + 1u < PRODUCT_SLOTS ? slot + 1u : 0u;
        }
        return sum;
    }
    // CH products are fetched while CH are added, by turns (a batch of loads would hold the additions up); the barrier of a slot is
    // passed before the last ones of the slot before are added.
    constexpr int CH = 32;
    float4 v[2][CH / 4];
    uint32_t at = ptx::smem_u32(products) + lane * (PRODUCT_PITCH * 4u);
    auto load = [&](float4& to, int q) {
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(to.x), "=f"(to.y), "=f"(to.z), "=f"(to.w) : "r"(at + 16u * q) : "memory");
    };
    auto load_and_add = [&](int from) {
#pragma unroll
        for (int q = 0; q < CH / 4; ++q) {
            load(v[from ^ 1][q], q);
            sum = __fadd_rn(sum, v[from][q].x);
            sum = __fadd_rn(sum, v[from][q].y);
            sum = __fadd_rn(sum, v[from][q].z);
            sum = __fadd_rn(sum, v[from][q].w);
        }
    };
    barrier_sync(FULL);
#pragma unroll
    for (int q = 0; q < CH / 4; ++q) load(v[0][q], q);
#pragma unroll 1
    for (uint32_t k = 0; k < pieces; ++k) {
        at += CH * 4u;
        load_and_add(0);
        at += CH * 4u;
        load_and_add(1);
        at += CH * 4u;
        load_and_add(0);
        const uint32_t before = slot;
        slot = slot + 1u < PRODUCT_SLOTS ? slot + 1u : 0u;
        at = ptx::smem_u32(products + slot * SLOT) + lane * (PRODUCT_PITCH * 4u);
        if (k + 1u < pieces) barrier_sync(FULL + slot);
        if (k + PRODUCT_SLOTS < pieces) barrier_arrive(EMPTY + before);
        load_and_add(1);   // the last one fetches whatever lies there
    }
    return sum;
}
// The sums of N rows side by side (input i of row r at a[i * G + r]) over one piece, lane = output: sum + w[0] a[0] + ... in
// this order, every product and every sum rounded; the next granule of eight inputs is on its way while one is added.
// (mul.rn.f32x2 and add.rn.f32x2 were contracted to one fma.f32x2; a product as fma(x, y, -0.0) rounds the same and cannot be,
// if the compiler does not know the -0.0.)
template <int G, int N>
__device__ __forceinline__ void value_piece(float (&sum)[N], const uint8_t* piece, uint32_t tiles, uint32_t tile, const float* a, float minus_zero) {
    constexpr uint32_t GRANULES = PIECE / 8u;
    const uint32_t first = lane_granules(piece + tile * BOX_BYTES), second = first + tiles * BOX_BYTES;
    uint4 w[2];
    float x[2][8 * N];
    auto load = [&](int which, uint32_t g) {
        w[which] = granule(g < GRANULES / 2u ? first : second, g % 8u);
        const float* at = a + g * 8u * G;
        if (G == N) {
#pragma unroll
            for (int q = 0; q < 2 * N; ++q) {
                const float4 v = *reinterpret_cast<const float4*>(at + 4 * q);
                x[which][4 * q] = v.x; x[which][4 * q + 1] = v.y; x[which][4 * q + 2] = v.z; x[which][4 * q + 3] = v.w;
            }
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float2 v = *reinterpret_cast<const float2*>(at + e * G);
                x[which][N * e] = v.x; x[which][N * e + N - 1] = v.y;
            }
        }
    };
    auto add = [&](int b) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const uint32_t pair = e < 2 ? w[b].x : e < 4 ? w[b].y : e < 6 ? w[b].z : w[b].w;
            const float f = e & 1 ? high_half(pair) : low_half(pair);
            if (N == 1) {
                sum[0] = __fadd_rn(sum[0], __fmul_rn(f, x[b][e]));
            } else {
                const float2 s = add_pair(make_float2(sum[0], sum[N - 1]), fma_pair(make_float2(f, f), make_float2(x[b][N * e], x[b][N * e + N - 1]), make_float2(minus_zero, minus_zero)));
                sum[0] = s.x;
                sum[N - 1] = s.y;
            }
        }
    };
    load(0, 0u);
#pragma unroll 1
    for (uint32_t g = 0; g < GRANULES; g += VALUE_BODY) {
#pragma unroll
        for (uint32_t k = 0; k < VALUE_BODY; ++k) {
            load((k & 1u) ^ 1u, (g + k + 1u) % GRANULES);
            add(k & 1u);
        }
    }
}

// G: sequences of a cluster.  The shape follows from G and the channels of a CTA; it is the kernel's, since code that one shape does not
// need costs it instruction cache (32 sequences: 579 us per step, 590 with the others' in between).
//   BY_ROW: D has a warp per row and tile of outputs where that leaves no scheduler two of them, rather than two rows at once (16 sequences,
//     four rows of 32 outputs: 25 000 cycles, now 19 900; with eight warps, 64 sequences, 24 200 and 27 900)
//   WIDE: q, k and v of a channel are shared by two threads
enum StepShape { BY_ROW, PLAIN, WIDE };
__host__ __device__ constexpr StepShape step_shape(uint32_t group, uint32_t own) {
    return group == 1u ? PLAIN : own >= THREADS / 2u ? WIDE : group * (own / VALUE_OUT) <= WARPS / 2u ? BY_ROW : PLAIN;
}
template <int G, StepShape SHAPE>
__global__ void __launch_bounds__(THREADS, 1)
gen_step_kernel(const Step p) {
    extern __shared__ __align__(16) uint8_t step_smem[];
    __shared__ Layer layers[2];
    __shared__ Statistics stats;
    const uint32_t d = p.d, ffn = p.ffn, ctas = cluster_size(), rank = cluster_rank(), words = d / 32u;
    const uint32_t own = d / ctas, o0 = rank * own;                                  // channels of this CTA
    const uint32_t f_own = ffn / ctas, f0 = rank * f_own;                            // CMix hidden units
    const uint32_t v_own = (p.vocab + ctas - 1u) / ctas, v0 = min(rank * v_own, p.vocab), v_n = min(v_own, p.vocab - v0);
    const uint32_t pieces = ffn / PIECE, tiles = own / VALUE_OUT, stages = p.stages, stage_bytes = own * (PIECE * 2u);
    const bool staged = p.staged;                 // packed weights in shared memory
    const Layout at(G, d, ffn, ctas, stages, staged);
    constexpr int N = G < 2 ? 1 : 2;              // rows of a thread in D
    const bool alone = G * own == VALUE_OUT;      // D: one sum per lane of a warp
    uint8_t* const base = step_smem + (0u - ptx::smem_u32(step_smem)) % 1024u;   // the same in every CTA of the cluster
    uint8_t* ring = base + at.ring;
    float* products = reinterpret_cast<float*>(base + at.products);
    float* x = reinterpret_cast<float*>(base + at.rows);   // [G][d]
    float* in0 = x + G * d;                                     // [d][G]
    float* act = in0 + G * d;                                   // [ffn][G] in C and D, or [G][ffn] (act_by_row)
    float* in1 = act;                                           // [d][G], and the third input behind it, in A
    float* y = act + 2u * G * d;                                // [d][G] in A and B
    uint8_t* bits = base + at.bits;                             // [3][G][own]
    uint32_t* w_wide = reinterpret_cast<uint32_t*>(base + at.wide);
    uint32_t* w_o = reinterpret_cast<uint32_t*>(base + at.o);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    __shared__ Copies copies;
    const bool copier = warp == WARPS - 1u, issuer = copier && lane == 0u;   // its first lane asks for copies
    uint32_t layers_done = 0, heads_done = 0;     // phases of the barriers of the packed weights
    uint32_t slot = 0, lap = 0;                   // of the ring: the piece that is used next
    uint32_t fetch_slot = 0;                      // the piece that is fetched next
    // whether a barrier was told to expect something an odd number of times: of the ring and of the packed weights (by the issuer), of
    // the exchanges (by thread 0)
    uint32_t ring_odd = 0, packed_odd = 0, exchange_odd = 0;
    if (issuer) {
#pragma unroll 1
        for (uint32_t b = 0; b < BARS; ++b) ptx::mbar_init(copies.ring + b, b - MAX_STAGES < MAX_STAGES ? WARPS : 1u);
        ptx::fence_mbar_init();
        copies.gave_up = 0u;
    }
    cluster_arrive();
    cluster_wait();   // nobody is sent anything before
    auto load_layer = [&](uint32_t l) {
        const uint32_t* from = reinterpret_cast<const uint32_t*>(p.layers + l);
        uint32_t* to = reinterpret_cast<uint32_t*>(&layers[l & 1u]);
#pragma unroll 1
        for (uint32_t i = threadIdx.x; i < sizeof(Layer) / 4u; i += THREADS) to[i] = from[i];
    };
    const uint32_t own_bytes = own * words * 4u;
    auto fetch_qkv_o = [&](const Layer& L) {
        if (!issuer || !staged || has_given_up(copies)) return;
        packed_odd ^= 1u;
        ptx::mbar_arrive_expect_tx(copies.qkv_o(), 4u * own_bytes);
        for (uint32_t z = 0; z < 3u; ++z) copy_bytes(w_wide + z * own * words, L.qkv[z].bits + (size_t)o0 * words, own_bytes, copies.qkv_o());
        copy_bytes(w_o, L.o.bits + (size_t)o0 * words, own_bytes, copies.qkv_o());
    };
    // D takes its weights `passes` times: a warp has 32 outputs of N rows per pass
    auto fetch_piece = [&](uint32_t l, uint32_t i) {
        if (!issuer || has_given_up(copies)) return;
        ring_odd ^= 1u << fetch_slot;
        fetch_value(ring + fetch_slot * stage_bytes, p.values + l, o0, own, i % pieces * (PIECE / SLAB), PIECE / SLAB, copies.ring + fetch_slot);
        fetch_slot = fetch_slot + 1u < stages ? fetch_slot + 1u : 0u;
    };
    const uint32_t clusters = gridDim.x / ctas;
    for (uint32_t row = blockIdx.x / ctas * G; row < p.rows; row += clusters * G) {
        const uint32_t n = min((uint32_t)G, p.rows - row);
        load_layer(0);
#pragma unroll 1
        for (uint32_t r = 0; r < G; ++r) {   // embedding and ln0, which replaces it
            const uint16_t* e = p.embedding + (size_t)p.tokens[row + min(r, n - 1u)] * d;
#pragma unroll 1
            for (uint32_t c = threadIdx.x; c < d; c += THREADS) x[r * d + c] = h2f(e[c]);
        }
        __syncthreads();
        if (issuer && row < clusters * G) {   // the first rows: beside the sums, which are not this warp's (0.1 to 0.3 us a step)
#pragma unroll 1
            for (uint32_t l = 0; l < p.n_layers; ++l) ptx::tma_acquire_desc(p.values + l);
        }
        rows_statistics(x, in0, n, d, stats);
        __syncthreads();
        fetch_qkv_o(layers[0]);
#pragma unroll 1
        for (uint32_t c = threadIdx.x; c < d; c += THREADS) {
            const float w = h2f(p.ln0_w[c]), b = h2f(p.ln0_b[c]);
#pragma unroll 1
            for (uint32_t r = 0; r < n; ++r) x[r * d + c] = normalised(x[r * d + c], stats.mean[r], stats.inv[r], w, b);
        }
        // the pushes: `per` channels side by side of one row for a warp at a time
        uint32_t per = 1u;
        while (per < 32u && 2u * per <= n * min(own, 128u) / WARPS) per *= 2u;   // own is a multiple of 32
        const uint32_t sets = n * (own / per);
        auto push_set = [&](uint32_t l, uint32_t j, size_t& stream, uint32_t& r, uint32_t& c) {
            r = j / (own / per);
            c = j % (own / per) * per + lane;
            stream = ((size_t)l * p.rows + row + r) * d + o0 + c - lane;
            return lane < per && r < n;
        };
        auto push_begin = [&](uint32_t l) {   // of this warp's first set: asked for while something else is waited for
            size_t stream;
            uint32_t r, c;
            const bool live = push_set(l, warp, stream, r, c);
            return push::begin(p.push, stream, live, p.time);
        };
        push::Ahead ahead = push_begin(0u);
        constexpr bool act_by_row = SHAPE == BY_ROW;
        const uint32_t sums = act_by_row ? n * tiles : (n + N - 1u) / N * tiles, passes = (sums + WARPS - 1u) / WARPS, items = passes * pieces;   // of D
#pragma unroll 1
        for (uint32_t l = 0; l < p.n_layers; ++l) {
            const Layer& L = layers[l & 1u];   // everybody's since a barrier ago
#pragma unroll 1
            for (uint32_t stage = 0; stage < 3u; ++stage) {   // A, B, C
                const uint32_t n_out = stage == 0u ? 3u * own : stage == 1u ? own : f_own;
                if (stage != 1u) {
                    mixed_inputs<G>(p, L, l, stage / 2u, row, n, o0, own, x, in0, G * d);
                    if (staged) copies_wait(copies, stage ? copies.key() : copies.qkv_o(), layers_done, p, 0x602u);
                }
                __syncthreads();
                auto emit = [&](uint32_t o, uint32_t r, float v) {
                    if (stage == 0u) {
                        const uint32_t z = o / own, c = o - z * own;
                        bits[(z * G + r) * own + c] = v > 0.0f;   // src/rosa.rs:372-374
                    } else if (stage == 1u) {
                        x[r * d + o0 + o] = __fadd_rn(x[r * d + o0 + o], v);
                    } else {
                        const float m = fmaxf(v, 0.0f);           // src/model.rs:999
                        act[act_by_row ? r * ffn + f0 + o : (f0 + o) * G + r] = __fmul_rn(m, m);
                    }
                };
                // Q, K and V of this CTA's channels from matrix z0 on, J of them and all rows per thread.
                auto qkv_of_channels = [&](auto matrices, uint32_t z0, uint32_t thread, uint32_t threads) {
                    constexpr int J = decltype(matrices)::value;
#pragma unroll 1
                    for (uint32_t c = thread; c < own; c += threads) {
                        uint32_t scale[J], bias[J];
#pragma unroll
                        for (int z = 0; z < J; ++z) {
                            scale[z] = load_half_ahead(L.qkv[z0 + z].scale + o0 + c);
                            bias[z] = load_half_ahead(L.qkv[z0 + z].bias + o0 + c);
                        }
                        float sum[J][G];
                        packed_sums<G, J, true>(in0 + z0 * (G * d), G * d, w_wide + (z0 * own + c) * words, own * words, d, sum);
#pragma unroll
                        for (int z = 0; z < J; ++z)
#pragma unroll
                            for (int r = 0; r < G; ++r)
                                if (r < n) emit((z0 + z) * own + c, r, __fadd_rn(low_half(bias[z]), __fmul_rn(low_half(scale[z]), sum[z][r])));
                    }
                };
                // As many outputs per thread as leave two warps for every scheduler, since one by itself issues every other cycle at best
                // (64 sequences, 128 channels and 512 hidden units of a CTA: q, k and v of a channel by one thread 12 400 cycles, q and k beside v
                // 11 400; four hidden units per thread 14 000, two 12 700).
                if (SHAPE == WIDE && stage == 0u && staged) {
                    if (threadIdx.x < THREADS / 2u) qkv_of_channels(std::integral_constant<int, 2>{}, 0u, threadIdx.x, THREADS / 2u);
                    else qkv_of_channels(std::integral_constant<int, 1>{}, 2u, threadIdx.x - THREADS / 2u, THREADS / 2u);
                } else if (stage == 2u && n_out >= 4u * THREADS) {
                    packed_outputs<G, 4>(L.key, staged ? w_wide : L.key.bits + (size_t)f0 * words, in0, n, d, f0, n_out, emit);
                } else if (stage == 2u && n_out >= THREADS && n_out % 2u == 0u) {
                    packed_outputs<G, 2>(L.key, staged ? w_wide : L.key.bits + (size_t)f0 * words, in0, n, d, f0, n_out, emit);
                } else {
#pragma unroll 1
                    for (uint32_t o = threadIdx.x; o < n_out; o += THREADS) {
                        const uint32_t z = stage == 0u ? o / own : 0u, first = stage == 2u ? f0 : o0, k = o - z * own;
                        const Packed& P = stage == 0u ? L.qkv[z] : stage == 1u ? L.o : L.key;
                        const uint32_t scale = load_half_ahead(P.scale + first + k), bias = P.bias ? load_half_ahead(P.bias + first + k) : 0u;
                        const uint32_t* w = staged ? (stage == 1u ? w_o : w_wide) + (size_t)o * words : P.bits + (size_t)(first + k) * words;
                        float sum[1][G];
                        packed_sums<G, 1, false>(stage == 1u ? y : in0 + z * (G * d), 0u, w, 0u, d, sum);
#pragma unroll
                        for (int r = 0; r < G; ++r)
                            if (r < n) emit(o, r, __fadd_rn(low_half(bias), __fmul_rn(low_half(scale), sum[0][r])));
                    }
                }
                __syncthreads();
                if (stage == 0u) {
#pragma unroll 1
                    for (uint32_t j = warp; j < sets; j += WARPS) {
                        size_t stream;
                        uint32_t r, c;
                        const bool live = push_set(l, j, stream, r, c);
                        uint32_t e = 0;
                        if (live) e = load_half_ahead(L.e + o0 + c);
                        if (j != warp) ahead = push::begin(p.push, stream, live, p.time);
                        const uint8_t* b = bits + r * own + c;
                        const bool idx = push::step(p.push, stream, live, p.time, ahead, live ? b[0] : 0u, live ? b[G * own] : 0u, live ? b[2 * G * own] : 0u);
                        if (live) y[(o0 + c) * G + r] = idx ? low_half(e) : -low_half(e);   // src/model.rs:1344-1351
                    }
                    __syncthreads();
                }
                const bool in_rows = stage == 1u || (stage == 2u && act_by_row);
                const float* shared_out = stage == 0u ? y + o0 * G : stage == 1u ? x + o0 : act + (act_by_row ? f0 : f0 * G);
                const bool sent = send_to_cluster(shared_out, in_rows ? n : 1u, stage == 1u ? d : ffn, (stage == 2u ? f_own : own) * (in_rows ? 1u : G), copies,
                                                  copies.exchange(stage));
                if (sent) exchange_odd ^= 1u << stage;
                if (stage == 0u) {
                    // the key weights, in place of Q, K and V, and the first pieces of D
                    if (issuer && staged && !has_given_up(copies)) {
                        packed_odd ^= 2u;
                        ptx::mbar_arrive_expect_tx(copies.key(), f_own * words * 4u);
                        copy_bytes(w_wide, L.key.bits + (size_t)f0 * words, f_own * words * 4u, copies.key());
                    }
                    if (!alone) {
#pragma unroll 1
                        for (uint32_t i = 0; i < min(items, stages - 1u); ++i) fetch_piece(l, i);
                    } else if (issuer && !has_given_up(copies)) {
                        ring_odd ^= 1u;
                        fetch_value(ring, p.values + l, o0, own, 0u, ffn / SLAB, copies.ring);
                    }
                } else if (stage == 2u && l + 1u < p.n_layers) {
                    load_layer(l + 1u);
                }
                copies_wait(copies, copies.exchange(stage), layers_done, p, 0x607u);
            }
            // ---- D
            if (alone) {
                const float sum = value_alone(ring, copies, lap, act, pieces, products, p);
                if (warp == 0u) x[o0 + lane] = __fadd_rn(x[o0 + lane], sum);
                ++lap;
            } else {
#pragma unroll 1
                for (uint32_t pass = 0, i = 0; pass < passes; ++pass) {
                    const uint32_t mine = pass * WARPS + warp, tile = mine % tiles, pair = mine / tiles;
                    float sum[N];
#pragma unroll
                    for (int r = 0; r < N; ++r) sum[r] = 0.0f;
#pragma unroll 1
                    for (uint32_t k = 0; k < pieces; ++k, ++i) {
                        if (copier && i + stages - 1u < items) {   // into the place of the piece before this one
                            if (i) copies_wait(copies, copies.empty() + (slot ? slot : stages) - 1u, slot ? lap : lap - 1u, p, 0x606u);
                            fetch_piece(l, i + stages - 1u);
                        }
                        copies_wait(copies, copies.ring + slot, lap, p, 0x604u);
                        if (mine < sums) {
                            const uint8_t* piece = ring + slot * stage_bytes;
                            if constexpr (act_by_row) {
                                float one[1] = {sum[0]};
                                value_piece<1, 1>(one, piece, tiles, tile, act + pair * ffn + k * PIECE, p.minus_zero);
                                sum[0] = one[0];
                            } else {
                                value_piece<G, N>(sum, piece, tiles, tile, act + k * PIECE * G + pair * N, p.minus_zero);
                            }
                        }
                        __syncwarp();
                        if (lane == 0u) ptx::mbar_arrive(copies.empty() + slot);
                        if (++slot == stages) { slot = 0; ++lap; }
                    }
                    if (mine < sums) {
#pragma unroll
                        for (int r = 0; r < N; ++r)
                            if (act_by_row ? r == 0 : pair * N + r < n) {
                                float* to = x + (act_by_row ? pair : pair * N + r) * d + o0 + tile * VALUE_OUT + lane;
                                *to = __fadd_rn(*to, sum[r]);
                            }
                    }
                }
            }
            ++layers_done;
            __syncthreads();
            if (send_to_cluster(x + o0, n, d, own, copies, copies.exchange(3u))) {
                exchange_odd ^= 8u;
            } else if (threadIdx.x < ctas) {   // the others need not wait for what is not sent
                asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(ptx::cluster_map(&copies.gave_up, threadIdx.x)),
                             "r"(*static_cast<volatile uint32_t*>(&copies.gave_up)) : "memory");
            }
            if (l + 1u < p.n_layers) {
                fetch_qkv_o(layers[(l + 1u) & 1u]);
                ahead = push_begin(l + 1u);
            }
            copies_wait(copies, copies.exchange(3u), layers_done - 1u, p, 0x608u);
        }
        // The head: its weights by as many outputs at a time as the ring has room for, where they lie on 16-byte borders.
        const bool head_staged = staged && v_own * words % 4u == 0u && v_n * words % 4u == 0u;
        const uint32_t chunk = head_staged ? max(stages * stage_bytes / (words * 4u) / 4u * 4u, 4u) : max(v_n, 1u);
        auto fetch_head = [&](uint32_t from) {
            if (!issuer || !head_staged || has_given_up(copies)) return;
            packed_odd ^= 4u;
            const uint32_t bytes = min(chunk, v_n - from) * words * 4u;
            ptx::mbar_arrive_expect_tx(copies.head(), bytes);
            copy_bytes(ring, p.head.bits + (size_t)(v0 + from) * words, bytes, copies.head());
        };
        if (v_n) fetch_head(0u);
        rows_statistics(x, in0, n, d, stats);
        __syncthreads();
#pragma unroll 1
        for (uint32_t c = threadIdx.x; c < d; c += THREADS) {
            const float w = h2f(p.ln_out_w[c]), b = h2f(p.ln_out_b[c]);
            for (uint32_t r = 0; r < G; ++r) in1[c * G + r] = r < n ? normalised(x[r * d + c], stats.mean[r], stats.inv[r], w, b) : 0.0f;
        }
        auto emit = [&](uint32_t o, uint32_t r, float v) { p.logits[(size_t)(row + r) * p.vocab + v0 + o] = v; };
#pragma unroll 1
        for (uint32_t from = 0; from < v_n; from += chunk) {
            if (from) {
                __syncthreads();
                fetch_head(from);
            }
            if (head_staged) copies_wait(copies, copies.head(), heads_done++, p, 0x605u);
            __syncthreads();
            const uint32_t* w = head_staged ? reinterpret_cast<const uint32_t*>(ring) : p.head.bits + (size_t)v0 * words;
            const uint32_t outputs = min(chunk, v_n - from);
            auto out = [&](uint32_t o, uint32_t r, float v) { emit(from + o, r, v); };
            if (outputs % 4u == 0u) packed_outputs<G, 4>(p.head, w, in1, n, d, v0 + from, outputs, out);
            else packed_outputs<G, 1>(p.head, w, in1, n, d, v0 + from, outputs, out);
        }
        cluster_arrive();
        cluster_wait();   // the rows are written anew only when nobody reads them
    }
    // After a give-up, copies and shares may still be on their way into this CTA's shared memory: it waits for those that its
    // barriers expect (a phase that is over is passed at once), and a while for shares that came without being expected.
    if (has_given_up(copies)) {
        constexpr uint32_t DRAIN = 1u << 12;
        if (issuer) {
#pragma unroll 1
            for (uint32_t b = 0; b < stages; ++b) ptx::mbar_wait(copies.ring + b, ~(ring_odd >> b) & 1u, DRAIN);
#pragma unroll 1
            for (uint32_t b = 0; b < 3u; ++b) ptx::mbar_wait(copies.qkv_o() + b, ~(packed_odd >> b) & 1u, DRAIN);
        }
        if (threadIdx.x == 0u) {
            *static_cast<volatile uint32_t*>(p.status) = ULLIS_DEV_WAIT_TIMEOUT;
            *static_cast<volatile uint32_t*>(p.status + 1) = copies.gave_up;
#pragma unroll 1
            for (uint32_t b = 0; b < 4u; ++b) ptx::mbar_wait(copies.exchange(b), ~(exchange_odd >> b) & 1u, DRAIN);
#pragma unroll 1
            for (uint32_t i = 0; i < 64u; ++i) __nanosleep(1000);
        }
    }
    __syncthreads();
}

}  // namespace gen
}  // namespace ullis
