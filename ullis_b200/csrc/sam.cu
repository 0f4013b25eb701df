// ROSA 1-bit match on the GPU, bit streams read and idx bits written as
// stream-major 32-step words; results equal T pushes of the reference's
// RosaSam (src/rosa.rs:100-176) for every stream.
//
// Up to 8192 steps a stream needs no automaton (rosa_match below): every step
// is looked up by itself (rosa_heads.cuh, rosa_context.cuh) or in sets of lags
// (rosa_match.cuh), so no launch lasts as long as a stream's chain of steps.
// 64 sequences x 512 channels x 2048 steps: 0.85 ms on evenly spread bits where
// the automaton took 11.3, 0.60 against 2.10 per layer of the benchmark model;
// 1 sequence 0.07 against 0.62.
//
// Longer streams, and calls that ask for one of its forms, run the suffix
// automaton: one thread per (sequence, channel) stream, automaton state in a
// per-stream block of global scratch (compact 16-bit state ids whenever
// 2T+2 <= 65535).  The per-stream algorithm lives in sam_core.cuh.  Streams
// with constant k bits are finished by a closed form first; the rest are
// processed in waves sized to the scratch budget, so any batch works; all
// waves are enqueued back to back on the runtime stream.
#include <algorithm>

#include "kernels.hpp"
#include "rosa_context.cuh"
#include "rosa_heads.cuh"
#include "rosa_match.cuh"
#include "sam_coop.cuh"
#include "sam_core.cuh"

namespace ullis {
namespace k {

namespace {

// Streams that need no automaton are settled here with a few word operations
// (sam_core.cuh, "constant k", "constant v" and "constant q"): k bits all equal, v bits all 0
// (idx = 0), v bits all 1 (idx_t = "q_t has occurred among the earlier keys") and q bits all
// equal (a scan over the key runs, in a kernel of its own).
// Every other stream id is appended to `list` for the automaton kernels.
// Eight lanes share a stream: each takes every eighth word of its three bit streams (a group reads 32
// consecutive bytes per request), the group combines by shuffle, and the closed forms - all of them word by
// word - are written the same way.  One thread per stream spent its time in 3 x 64 dependent strided loads.
constexpr int CLASSIFY_LANES = 8;
// COUNT_UNEVEN: how many of the listed streams have walks of more than UNEVEN_PER_ROW positions per row along their runs alone
// (rosa_heads.cuh; T <= 2048).
constexpr uint32_t UNEVEN_PER_ROW = 10, UNEVEN_SHARE = 16;
template <bool COUNT_UNEVEN>
__global__ void __launch_bounds__(128)
rosa_classify_kernel(const uint32_t* __restrict__ q_sw, const uint32_t* __restrict__ k_sw,
                     const uint32_t* __restrict__ v_sw, uint32_t* __restrict__ idx_sw, size_t streams, uint32_t T,
                     size_t wps, uint32_t* __restrict__ list, uint32_t* __restrict__ count,
                     uint32_t* __restrict__ cq_list, uint32_t* __restrict__ cq_count, uint32_t* __restrict__ given_up,
                     uint32_t* __restrict__ uneven_count) {
    chain_entry();
    constexpr uint32_t G = CLASSIFY_LANES;
    const size_t s = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
    if (s >= streams) return;   // a whole group
    if (given_up && threadIdx.x % G == 0) given_up[s] = 0u;
    const uint32_t sub = threadIdx.x % G, lane = threadIdx.x & 31u;
    const uint32_t group = ((1u << G) - 1u) << (lane & ~(G - 1u));
    const uint32_t* qw = q_sw + s * wps;
    const uint32_t* kw = k_sw + s * wps;
    const uint32_t* vw = v_sw + s * wps;
    uint32_t* out = idx_sw + s * wps;
    const uint32_t last = (uint32_t)wps - 1u;
    const uint32_t tail = (T & 31u) ? ((1u << (T & 31u)) - 1u) : 0xFFFFFFFFu;
    // AND and OR of the three streams over steps 0 .. T-1 (the bits past T in the last word count for neither)
    uint32_t all[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, any[3] = {0u, 0u, 0u};
    uint32_t keys = 0, rows = 0;   // in runs of ones, and of zeros << 16: positions of keys, and words with a query
    for (uint32_t w = sub; w <= last; w += G) {
        const uint32_t m = w == last ? tail : 0xFFFFFFFFu;
        const uint32_t x[3] = {kw[w], vw[w], qw[w]};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            all[a] &= x[a] | ~m;
            any[a] |= x[a] & m;
        }
        if (COUNT_UNEVEN) {
            keys += (uint32_t)__popc(heads::ends_of_runs(x[0] & m)) + ((uint32_t)__popc(heads::ends_of_runs(~x[0] & m)) << 16);
            rows += (heads::ends_of_runs(x[2] & m) ? 1u : 0u) + (heads::ends_of_runs(~x[2] & m) ? 0x10000u : 0u);
        }
    }
    bool uneven = false;
    if (COUNT_UNEVEN) {
#pragma unroll
        for (uint32_t o = 1; o < G; o <<= 1) {
            keys += __shfl_xor_sync(group, keys, o);
            rows += __shfl_xor_sync(group, rows, o);
        }
        const uint32_t most = UNEVEN_PER_ROW * (last + 1u);
        uneven = heads::walks_too_long(keys & 0xFFFFu, rows & 0xFFFFu, most) || heads::walks_too_long(keys >> 16, rows >> 16, most);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (uint32_t o = 1; o < G; o <<= 1) {
            all[a] &= __shfl_xor_sync(group, all[a], o);
            any[a] |= __shfl_xor_sync(group, any[a], o);
        }
    }
    auto constant = [&](int a, uint32_t* c) {
        if (all[a] == 0xFFFFFFFFu) { *c = 1u; return true; }
        if (any[a] == 0u) { *c = 0u; return true; }
        return false;
    };
    uint32_t c = 0;
    if (constant(0, &c)) {
        // sam::run_constant_k, a word per lane
        for (uint32_t w = sub; w <= last; w += G) {
            uint32_t word = (c ? qw[w] : ~qw[w]) & vw[w];
            if (w == 0) word &= ~1u;
            if (w == last) word &= tail;
            out[w] = word;
        }
    } else if (constant(1, &c)) {
        if (c == 0) {
            for (uint32_t w = sub; w <= last; w += G) out[w] = 0u;
        } else {
            // sam::run_constant_v_one: f = the first step whose key differs from k_0 (it exists: k is not constant)
            const uint32_t c0 = kw[0] & 1u, full = c0 ? 0xFFFFFFFFu : 0u;
            uint32_t f = T;
            for (uint32_t w = sub; w <= last && f == T; w += G) {
                uint32_t diff = kw[w] ^ full;
                if (w == last) diff &= tail;
                if (diff) f = w * 32u + (uint32_t)__ffs((int)diff) - 1u;
            }
#pragma unroll
            for (uint32_t o = 1; o < G; o <<= 1) f = min(f, __shfl_xor_sync(group, f, o));
            for (uint32_t w = sub; w <= last; w += G) {
                const uint32_t same = c0 ? qw[w] : ~qw[w];   // q_t == k_0
                uint32_t after;                               // bits of this word at steps > f
                if (f >= w * 32u + 31u) after = 0u;
                else if (f < w * 32u) after = 0xFFFFFFFFu;
                else after = ~((2u << (f - w * 32u)) - 1u);
                uint32_t word = (same & ~after) | after;
                if (w == 0) word &= ~1u;
                if (w == last) word &= tail;
                out[w] = word;
            }
        }
    } else if (sub == 0) {
        if (constant(2, &c)) cq_list[atomicAdd(cq_count, 1u)] = (uint32_t)s;   // constant q: a long scan, its own kernel
        else {
            list[atomicAdd(count, 1u)] = (uint32_t)s;
            if (COUNT_UNEVEN && uneven) atomicAdd(uneven_count, 1u);
        }
    }
}

// The constant-q streams listed by rosa_classify_kernel, one per thread: every thread of a warp runs the
// same scan (inside rosa_classify_kernel a warp would pay for it beside each of the shorter closed forms).
__global__ void __launch_bounds__(128)
rosa_constq_kernel(const uint32_t* __restrict__ q_sw, const uint32_t* __restrict__ k_sw, const uint32_t* __restrict__ v_sw,
                   uint32_t* __restrict__ idx_sw, uint32_t T, size_t wps, const uint32_t* __restrict__ cq_list,
                   const uint32_t* __restrict__ cq_count) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *cq_count) return;
    const size_t s = cq_list[i];
    sam::run_constant_q(q_sw[s * wps] & 1u, k_sw + s * wps, v_sw + s * wps, idx_sw + s * wps, T);
}

// Only `lanes` threads of each warp carry a stream (the others exit at once).
// A warp-level load completes when its slowest lane does, and a stream's
// accesses are pointer chases into its own state block, so fewer streams per
// warp (and more warps) shortens every dependent step.  Work item i of this
// launch is stream list[first + i]; its state block is block i of `scratch`.
template <typename Ix, int ALGO>
__global__ void __launch_bounds__(128)
rosa_sam_kernel(uint8_t* __restrict__ scratch, size_t scratch_stride, const uint32_t* __restrict__ q_sw,
                const uint32_t* __restrict__ k_sw, const uint32_t* __restrict__ v_sw,
                uint32_t* __restrict__ idx_sw, const uint32_t* __restrict__ list,
                const uint32_t* __restrict__ count, size_t first, size_t wave, uint32_t T, size_t wps, int lanes,
                uint32_t* __restrict__ status) {
    const int lane = threadIdx.x & 31;
    const int spread = 32 / lanes;
    if (lane % spread != 0) return;
    const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const size_t item = warp * lanes + lane / spread;
    // the grid is rounded up to whole CTAs: an item past the wave has no state block (it belongs to the next wave)
    if (item >= wave || first + item >= *count) return;
    const size_t s = list[first + item];
    uint8_t* block = scratch + item * scratch_stride;
    const uint32_t* qw = q_sw + s * wps;
    const uint32_t* kw = k_sw + s * wps;
    const uint32_t* vw = v_sw + s * wps;
    uint32_t* out = idx_sw + s * wps;
    if (ALGO == ULLIS_CUDA_SAM_EAGER)
        sam::run_eager<Ix>(block, qw, kw, vw, out, T, nullptr);
    else if (!sam::run_euler<Ix>(block, qw, kw, vw, out, T, nullptr)) {
        if (atomicCAS(status, ULLIS_DEV_OK, ULLIS_DEV_SAM_CAPACITY) == ULLIS_DEV_OK) status[1] = (uint32_t)s;
    }
}

// streams of the wave [first, first + wave) that reached the automaton
__device__ __forceinline__ uint32_t wave_items(uint32_t total, size_t first, size_t wave) {
    if (first >= total) return 0u;
    const size_t left = total - first;
    return (uint32_t)(left < wave ? left : wave);
}

// Two-kernel form of the O(T log T) schedule for streams whose tour / pass 2
// working set fits shared memory: pass 1 one thread per stream (below), then
// one warp per stream for the parallel phases (sam_coop.cuh).
// WORDS: 0 = field-wise state layout, 1 = packed words, 2 = packed words with the climb left to the tour kernel,
// 3 = the same without the register copy of the query state's words (one load per step instead of the patches)
// (a kernel each, so that the form that runs gets the registers to itself)
// (16 CTAs per SM = 32 registers: with 40 registers the same loop ran 4 % slower at 64 sequences and 40 % slower at 8)
template <int WORDS>
__global__ void __launch_bounds__(128, 16)
rosa_pass1_kernel(uint8_t* __restrict__ scratch, size_t scratch_stride, const uint32_t* __restrict__ q_sw,
                  const uint32_t* __restrict__ k_sw, const uint32_t* __restrict__ list,
                  const uint32_t* __restrict__ count, size_t first, size_t wave, uint32_t T, size_t wps, int lanes,
                  uint32_t dense_count, uint32_t sparse_count, uint32_t* __restrict__ hint) {
    // how many streams reached the automaton, for the host's choice of kernel the next time round (see rosa_sam)
    if (hint && blockIdx.x == 0 && threadIdx.x == 0) *hint = *count;
    // lanes == 0: choose from the number of streams that are left, which only the device knows -
    // many streams: four per warp (fewer issued instructions); fewer: two, then one per warp (more
    // warps to hide the pointer-chase latency).  The grid is sized for one per warp.
    if (lanes == 0) lanes = *count > dense_count ? 4 : *count > sparse_count ? 2 : 1;
    const int lane = threadIdx.x & 31;
    const int spread = 32 / lanes;
    if (lane % spread != 0) return;
    const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const size_t item = warp * lanes + lane / spread;
    // the grid is sized for one stream per warp and rounded up to whole CTAs: with several streams per warp an
    // item can lie past the wave, where it has no state block (it belongs to the next wave)
    if (item >= wave || first + item >= *count) return;
    const size_t s = list[first + item];
    sam::EulerBlock<uint16_t> B(scratch + item * scratch_stride, T);
    if (WORDS == 3) sam::euler_pass1_words<true, true>(B, q_sw + s * wps, k_sw + s * wps, T);
    else if (WORDS == 2) sam::euler_pass1_words<true, false>(B, q_sw + s * wps, k_sw + s * wps, T);
    else if (WORDS == 1) sam::euler_pass1_words<false>(B, q_sw + s * wps, k_sw + s * wps, T);
    else sam::euler_pass1<uint16_t>(B, q_sw + s * wps, k_sw + s * wps, T, nullptr);
}

// The same serial pass with the state array of the stream in shared memory, for calls with so few streams that
// every one of them gets its own one-warp CTA at once (six per SM at T = 2048): lane 0 runs the loop - a state
// visit is then a shared-memory access instead of a trip through L1, whose lines the step's own stores keep
// displacing - and the whole warp copies the states out for the tour kernel.  The grid covers every stream of
// the wave, so any number of them is handled (in rounds of resident CTAs); the host launches this form only
// when it expects one round.
__global__ void __launch_bounds__(32)
rosa_pass1_smem_kernel(uint8_t* __restrict__ scratch, size_t scratch_stride, const uint32_t* __restrict__ q_sw,
                       const uint32_t* __restrict__ k_sw, const uint32_t* __restrict__ list,
                       const uint32_t* __restrict__ count, size_t first, size_t wave, uint32_t T, size_t wps,
                       uint32_t* __restrict__ hint) {
    extern __shared__ __align__(16) uint8_t pass1_states[];
    if (hint && blockIdx.x == 0 && threadIdx.x == 0) *hint = *count;
    const size_t item = blockIdx.x;
    if (item >= wave_items(*count, first, wave)) return;
    const size_t s = list[first + item];
    sam::EulerBlock<uint16_t> B(scratch + item * scratch_stride, T);
    if (threadIdx.x == 0) {
        sam::EulerBlock<uint16_t> S = B;
        S.N = reinterpret_cast<sam::Node<uint16_t>*>(pass1_states);
        sam::euler_pass1_words<true, true>(S, q_sw + s * wps, k_sw + s * wps, T);
    }
    __syncwarp();
    const uint32_t n = B.meta[0];   // written by lane 0 just now
    const uint4* src = reinterpret_cast<const uint4*>(pass1_states);
    uint4* dst = reinterpret_cast<uint4*>(B.N);
    for (uint32_t i = threadIdx.x; i < (n + 1u) / 2u; i += 32u) dst[i] = src[i];
}

// Pass 1 in three parts (sam_core.cuh, "pass 1 in three parts"): the extend chain and the query walk as two
// kernels with one thread per stream each, the climb inside the tour kernel.  Work items and state blocks as in
// rosa_pass1_kernel.
__device__ __forceinline__ bool split_item(const uint32_t* __restrict__ count, size_t first, size_t wave, int lanes,
                                           uint32_t dense_count, uint32_t sparse_count, size_t* item_out) {
    if (lanes == 0) lanes = *count > dense_count ? 4 : *count > sparse_count ? 2 : 1;
    const int lane = threadIdx.x & 31;
    const int spread = 32 / lanes;
    if (lane % spread != 0) return false;
    const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const size_t item = warp * lanes + lane / spread;
    if (item >= wave || first + item >= *count) return false;
    *item_out = item;
    return true;
}

__global__ void __launch_bounds__(128, 16)
rosa_extend_kernel(uint8_t* __restrict__ scratch, size_t scratch_stride, const uint32_t* __restrict__ k_sw,
                   const uint32_t* __restrict__ list, const uint32_t* __restrict__ count, size_t first, size_t wave,
                   uint32_t T, size_t wps, int lanes, uint32_t dense_count, uint32_t sparse_count) {
    // All lanes of the group that belongs to a stream first fill the stream's `orig` array with NIL (16-byte
    // stores, the lanes side by side); then one lane of the group runs the chain and the others leave.
    if (lanes == 0) lanes = *count > dense_count ? 4 : *count > sparse_count ? 2 : 1;
    const int lane = threadIdx.x & 31, spread = 32 / lanes;
    const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const size_t item = warp * lanes + lane / spread;
    const bool live = item < wave && first + item < *count;
    if (live) {
        sam::EulerBlock<uint16_t> B(scratch + item * scratch_stride, T);
        uint4* o = reinterpret_cast<uint4*>(B.next);                       // 16-byte aligned by the layout
        const uint32_t vecs = (sam::node_capacity(T) * 2u + 15u) / 16u;    // the array's room is a multiple of 16 bytes
        for (uint32_t k = lane % spread; k < vecs; k += spread) o[k] = make_uint4(~0u, ~0u, ~0u, ~0u);
    }
    __syncwarp();
    if (!live || lane % spread != 0) return;
    const size_t s = list[first + item];
    sam::EulerBlock<uint16_t> B(scratch + item * scratch_stride, T);
    sam::euler_extend_words(B, k_sw + s * wps, T);
}

__global__ void __launch_bounds__(128, 16)
rosa_walk_kernel(uint8_t* __restrict__ scratch, size_t scratch_stride, const uint32_t* __restrict__ q_sw,
                 const uint32_t* __restrict__ list, const uint32_t* __restrict__ count, size_t first, size_t wave,
                 uint32_t T, size_t wps, int lanes, uint32_t dense_count, uint32_t sparse_count) {
    size_t item;
    if (!split_item(count, first, wave, lanes, dense_count, sparse_count, &item)) return;
    const size_t s = list[first + item];
    sam::EulerBlock<uint16_t> B(scratch + item * scratch_stride, T);
    uint32_t w = 0, h = 0;
    sam::euler_walk_words<false>(B, q_sw + s * wps, 0, T, w, h);
}

// The query walk with eight lanes per stream (sam_core.cuh euler_walk_chunked): each lane first walks an eighth of
// the steps from the guessed state "no match", all at once; then the pieces are put right one after the other,
// each from the true end state of the piece before it, which takes a few steps where matches are short.  Four
// streams per warp.  A lane only ever reads the records it wrote itself.
__global__ void __launch_bounds__(128, 16)
rosa_walk_chunked_kernel(uint8_t* __restrict__ scratch, size_t scratch_stride, const uint32_t* __restrict__ q_sw,
                         const uint32_t* __restrict__ list, const uint32_t* __restrict__ count, size_t first, size_t wave,
                         uint32_t T, size_t wps) {
    const int lane = threadIdx.x & 31, group = lane >> 3, c = lane & 7;
    const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const size_t item = warp * 4 + group;
    if (item >= wave || first + item >= *count) return;   // the eight lanes of a group leave together
    const size_t s = list[first + item];
    sam::EulerBlock<uint16_t> B(scratch + item * scratch_stride, T);
    const uint32_t* qw = q_sw + s * wps;
    const uint32_t piece = (((T + 7u) >> 3) + 31u) & ~31u;
    const uint32_t t0 = min((uint32_t)c * piece, T), t1 = min(t0 + piece, T);
    uint32_t w = 0, h = 0;
    sam::euler_walk_words<false>(B, qw, t0, t1, w, h);
    const unsigned mask = 0xFFu << (8 * group);
    for (int k = 1; k < 8; ++k) {
        const uint32_t pw = __shfl_sync(mask, w, (lane & ~7) + k - 1), ph = __shfl_sync(mask, h, (lane & ~7) + k - 1);
        if (c != k) continue;
        if (t0 >= t1) {           // an empty piece hands the state on
            w = pw; h = ph;
        } else {
            uint32_t tw = pw, th = ph;
            if (sam::euler_walk_words<true>(B, qw, t0, t1, tw, th) == t1) { w = tw; h = th; }   // never met: its own end state
        }
    }
}

template <int NT, int MODE = 0>   // 0: pass 1 left v_t; 1: split form (climb here, clones from orig); 2: deferred climb
__global__ void __launch_bounds__(NT)
rosa_coop_kernel(uint8_t* __restrict__ scratch, size_t scratch_stride, const uint32_t* __restrict__ v_sw,
                 uint32_t* __restrict__ idx_sw, const uint32_t* __restrict__ list, const uint32_t* __restrict__ count,
                 size_t first, uint32_t T, size_t wps, uint32_t* __restrict__ status) {
    extern __shared__ __align__(16) uint8_t coop_smem[];
    const size_t item = blockIdx.x;
    if (first + item >= *count) return;
    const size_t s = list[first + item];
    sam::EulerBlock<uint16_t> B(scratch + item * scratch_stride, T);
    if (B.meta[0] > sam::node_capacity(T)) {  // cannot happen: at most 2T states
        if (threadIdx.x == 0 && atomicCAS(status, ULLIS_DEV_OK, ULLIS_DEV_SAM_CAPACITY) == ULLIS_DEV_OK)
            status[1] = (uint32_t)s;
        return;
    }
    sam::coop_tour_pass2<NT, MODE != 0, MODE == 1>(coop_smem, B, v_sw + s * wps, idx_sw + s * wps, T);
}

// The listed streams by contexts (rosa_context.cuh), a CTA per stream, CTAs take streams from a counter until they run
// out.  A stream whose buckets are too large, or whose agreements turn out to be long, goes to `hard` instead.
// (step, key position in its bucket) pairs per step: up to which a stream is taken by its last bits without looking at
// the other way, and up to which at all.
struct ContextLimits {
    uint32_t easy, by_bits, by_runs;
    // 32-step comparisons beyond the first, and words gone back, per thread before a stream is given up
    uint32_t deep_by_bits, deep_by_runs;
};

// Where less than half of the CTAs would have a stream, two or more take one: each sorts all of its keys and answers its share of the
// steps (one sequence of the default model with gain N(0, 0.02), 64 of 512 streams listed, 148 CTAs: the slowest stream 130 000 cycles,
// 22 000 of them for the sort).
constexpr uint32_t MAX_PARTS = 4, PARTS_MAX_STREAMS = 4;   // per SM: of more hardly ever so few are listed, and the form costs the others 3 %
constexpr uint32_t CONTEXT_LARGE = 48;   // positions before a step in its buckets from which on the whole warp looks through them

struct ContextLayout {   // bytes of shared memory
    uint32_t hist, start, q, k, v, q_ends, k_ends, in_word, before, out, entries, steps, total;   // for up to c bits
    __host__ __device__ ContextLayout(uint32_t T, uint32_t c, uint32_t warps) {
        const uint32_t C = 1u << c, words = (T + 31u) / 32u + 1u;
        entries = 0;                           // Entry [T]
        hist = entries + T * 8u;               // u16 [warps][C]: counts, then write positions; behind them [C] for the steps
        start = hist + (warps + 1u) * C * 2u;  // u16 [C + 2]
        q = start + (C + 2u) * 2u;
        k = q + words * 4u;
        v = k + words * 4u;
        before = v + words * 4u;               // u32 [2][words]
        out = before + words * 8u;
        in_word = out + words * 4u;             // u16 [2][words]
        q_ends = in_word + words * 4u;         // u16 [words]
        k_ends = q_ends + words * 2u;
        steps = k_ends + words * 2u;           // u16 [T]
        total = (steps + T * 2u + 15u) & ~15u;
    }
};

// Bits of the longest contexts of a shape.
__host__ __device__ inline uint32_t context_bits(uint32_t T, bool together) { return together ? context::bits_for_uneven(T) : context::bits_for(T); }

// The streams whose keys are spread evenly (rosa_heads.cuh).  A stream is cut into `pieces`, a warp takes one: it puts the keys
// of the rows before into tables of its own and goes on from there.  The other streams go to `left`, once: a stream is given up
// as soon as the walks of a piece, the longest of each row, have come to more than `base` + `per_row` positions per row so far, 32
// steps beyond the first window counted as a position.  given_up: a word per stream, zero before (2: to rosa_match_kernel).
struct HeadsLayout {   // bytes of shared memory of a warp
    uint32_t latest_7, latest_3, link, q, k, v, total;   // latest_11 is at 0
    __host__ __device__ explicit HeadsLayout(uint32_t T) {
        const uint32_t words = (T + 31u) / 32u;
        latest_7 = heads::LATEST_11 * 2u;
        latest_3 = latest_7 + heads::LATEST_7 * 4u;
        link = latest_3 + heads::LATEST_3 * 4u;   // u16 [32 * words + 2]: by position + 1, the latest one before it with its context
        q = link + (32u * words + 2u) * 2u;       // u32 [words + 1]
        k = q + (words + 1u) * 4u;
        v = k + (words + 1u) * 4u;                // u32 [words]
        total = (v + words * 4u + 15u) & ~15u;
    }
};

struct HeadsCall {
    uint32_t warps;   // of a CTA that take pieces: as many as have room in its shared memory
    uint32_t pieces, base, per_row;
    uint32_t *next, *left, *left_count, *given_up;
    const uint32_t* uneven_count;
};

// A piece is left out, or its walk broken off, when another one has given the stream up; and a stream whose runs alone make its walks too long,
// `base` + RUNS_PER_ROW positions per row, is given up before its keys are put in.  (Without either every piece of an uneven stream spent its
// own `base` and more.  us of the ROSA kernels, contexts alone / before / now: 16 x 2048 steps x 512 channels, bits of probability 0.9 2112 / 2340 /
// 2135, of slow changes 1099 / 1302 / 1127, of clean periods 1343 / 1650 / 1509; 5 x 2048 725 / 877 / 741, 401 / 553 / 418, 492 / 661 / 612; 4 x 700
// 171 / 286 / 180, 139 / 232 / 150, 260 / 277 / 279.  Whole calls in training: 16 x 2048 9.43 / 9.46 ms, 5 x 1531 3.25 / 3.25, 16 x 700 3.88 / 3.91.  With
// 12 per row more of those are given up, 24 leaves 4 x 700 of probability 0.9 at 277.)
constexpr uint32_t RUNS_PER_ROW = 16;

// Bound by the integer pipe: per row of 32 steps of the model's streams (2048 steps) about 350 warp instructions, 215 of them on
// that pipe, which takes one every second cycle - the refinement of the masks 100, the look-ups 70, the walk over the
// chains 70, the keys 40.  rosa_context_kernel sorts each stream first and compares what lies in a bucket: 750 per row.  Both kernels
// in all layers, gain 1 + N(0, 0.02), contexts alone before: default model 64 times 2048 steps 21.5 -> 12.8 ms, 16 5.8 -> 4.3, 8 3.2 -> 2.6,
// 64 times 512 6.5 -> 2.7, 16 times 700 2.4 -> 1.3.
__device__ __forceinline__ void heads_streams(const uint32_t* __restrict__ q_sw, const uint32_t* __restrict__ k_sw, const uint32_t* __restrict__ v_sw,
                                              uint32_t* __restrict__ idx_sw, const uint32_t* __restrict__ list, uint32_t total, uint32_t T, size_t wps,
                                              uint8_t* __restrict__ heads_mem, const HeadsCall& call) {
    constexpr uint32_t ALL = 0xFFFFFFFFu;
    const uint32_t words = (T + 31u) / 32u, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const HeadsLayout L(T);
    uint8_t* mem = heads_mem + warp * L.total;
    uint16_t* latest_11 = reinterpret_cast<uint16_t*>(mem);
    uint32_t* latest_7 = reinterpret_cast<uint32_t*>(mem + L.latest_7);
    uint32_t* latest_3 = reinterpret_cast<uint32_t*>(mem + L.latest_3);
    uint16_t* link = reinterpret_cast<uint16_t*>(mem + L.link);
    uint32_t* Q = reinterpret_cast<uint32_t*>(mem + L.q);
    uint32_t* K = reinterpret_cast<uint32_t*>(mem + L.k);
    uint32_t* V = reinterpret_cast<uint32_t*>(mem + L.v);
    if (warp >= call.warps) return;
    const uint32_t pieces = call.pieces, warps = gridDim.x * call.warps, above = ALL << lane << 1, below = (1u << lane) - 1u;
    const uint32_t piece_rows = heads::rows_of_piece(words, pieces);
    auto keys_in = [&](uint32_t row, uint32_t wk) {
        const uint32_t r1 = 32u * row + lane + 1u, ctx = wk >> 21;
        uint32_t before = latest_11[ctx];
        atomicMax(&latest_7[wk >> 25], r1);
        atomicMax(&latest_3[wk >> 29], r1);
        __syncwarp();   // the tables have been read
        latest_11[ctx] = (uint16_t)r1;
        __syncwarp();
        if (__any_sync(ALL, latest_11[ctx] != (uint16_t)r1)) {   // a context twice in the row: its last lane counts
            const uint32_t same = __match_any_sync(ALL, ctx);
            if (!(same & above)) latest_11[ctx] = (uint16_t)r1;
            if (same & below) before = heads::latest(row, same & below);
        }
        link[r1] = (uint16_t)before;
        __syncwarp();
    };
    auto give_up = [&](size_t s) {
        if (lane == 0u && atomicExch(&call.given_up[s], 1u) == 0u) call.left[atomicAdd(call.left_count, 1u)] = (uint32_t)s;
    };
    // The last pieces first, which have the most keys to put in.
    for (uint32_t item = warp * gridDim.x + blockIdx.x; item < total * pieces;
         item = warps + __shfl_sync(ALL, lane == 0u ? atomicAdd(call.next, 1u) : 0u, 0)) {
        const uint32_t piece = pieces - 1u - item / total;
        const size_t s = list[item % total], at = s * wps;
        const uint32_t row0 = min(piece * piece_rows, words), row1 = min(row0 + piece_rows, words);
        const uint32_t by_other = pieces > 1u && lane == 0u ? __ldcg(&call.given_up[s]) : 0u;
        const uint32_t most_along_runs = call.base + RUNS_PER_ROW * row1;
        uint32_t keys = 0;   // positions in runs of ones, and of zeros << 16
        __syncwarp();
        for (uint32_t w = lane; w < row1; w += 32u) {
            const uint32_t key = k_sw[at + w];
            Q[w + 1u] = q_sw[at + w];
            K[w + 1u] = key;
            V[w] = v_sw[at + w];
            keys += (uint32_t)__popc(heads::ends_of_runs(key)) + ((uint32_t)__popc(heads::ends_of_runs(~key)) << 16);
        }
        if (lane == 0u) Q[0] = K[0] = 0u;
        if (__any_sync(ALL, by_other)) continue;
        keys = __reduce_add_sync(ALL, keys);
        if (__any_sync(ALL, heads::walks_too_long(max(keys & 0xFFFFu, keys >> 16), row1, most_along_runs))) {
            uint32_t rows = 0;   // with a query in a run of ones, and of zeros << 16
            for (uint32_t w = lane; w < row1; w += 32u) {
                const uint32_t query = Q[w + 1u];
                rows += (heads::ends_of_runs(query) ? 1u : 0u) + (heads::ends_of_runs(~query) ? 0x10000u : 0u);
            }
            rows = __reduce_add_sync(ALL, rows);
            if (__any_sync(ALL, heads::walks_too_long(keys & 0xFFFFu, rows & 0xFFFFu, most_along_runs) || heads::walks_too_long(keys >> 16, rows >> 16, most_along_runs))) {
                give_up(s);
                continue;
            }
        }
        for (uint32_t i = lane; i < L.link / 16u; i += 32u) reinterpret_cast<uint4*>(mem)[i] = uint4{0u, 0u, 0u, 0u};
        __syncwarp();
        uint32_t k0 = 0u, q0 = Q[row0], work = 0;
        for (uint32_t row = 0; row < row0; ++row) {
            const uint32_t k1 = K[row + 1u];
            keys_in(row, __funnelshift_l(k0, k1, 31u - lane));
            k0 = k1;
        }
        bool gone = false;
        for (uint32_t row = row0; row < row1 && !gone; ++row) {
            const uint32_t k1 = K[row + 1u], q1 = Q[row + 1u], t = 32u * row + lane;
            const uint32_t wk = __funnelshift_l(k0, k1, 31u - lane), wq = __funnelshift_l(q0, q1, 31u - lane);
            uint32_t found = heads::probe_11(latest_11, wq);
            if (!found) found = heads::probe(latest_7, wq, 7u);
            if (!found) found = heads::probe(latest_3, wq, 3u);
            const uint32_t in_row = row ? heads::agreeing<false>(k0, k1, below, wq) : heads::agreeing<true>(k0, k1, below, wq);
            k0 = k1;
            q0 = q1;
            __syncwarp();
            keys_in(row, wk);
            // the latest lane of those that agree longest, and in how many bits
            const uint32_t near = heads::latest(row, in_row), near_key = __shfl_sync(ALL, wk, (near - 1u) & 31u);
            const uint32_t near_bits = min(min(context::leading(wq ^ near_key), heads::DEPTH), near);
            if (in_row && near_bits >= found >> 16) found = near_bits << 16 | near;
            const uint32_t most = call.base + call.per_row * (row - row0) - work;   // not below 0: the stream would be gone
            uint32_t r1 = found & 0xFFFFu, best = 0, walked = 0, p = found >> 16 == heads::DEPTH && t < T ? r1 : 0u;
            while (p && walked <= most) {
                uint32_t n = min(context::leading(wq ^ heads::window_before(K, p)), p);
                if (n == 32u) n = context::agreement(Q, K, t, p - 1u, 0u, walked);
                if (n > best) {
                    best = n;
                    r1 = p;
                }
                p = link[p];
                ++walked;
            }
            walked = __reduce_max_sync(ALL, walked);
            work += walked;
            gone = walked > most;
            if (walked > call.per_row && pieces > 1u) gone |= __any_sync(ALL, lane == 0u && __ldcg(&call.given_up[s]));
            const uint32_t word = __ballot_sync(ALL, r1 && t < T && (V[r1 >> 5] >> (r1 & 31u) & 1u));
            if (lane == 0u) idx_sw[at + row] = word;
        }
        if (gone) give_up(s);
    }
}

// TOGETHER: large buckets by a whole warp, one step after the other, and one bit more for the streams that are not easy (a stream
// at a time: default model with gain N(0, 0.02), contexts of 64 sequences 7.49 -> 6.97 ms, of one at 1000 steps 0.65 -> 0.54; with
// the bit for every stream of a launch even ones paid, 148 of 2048 steps 26 -> 34 us, of 4096 41 -> 55).  Runs where the
// number of listed streams is in [from, to).
// FORM: IN_PARTS costs the other calls 3 % of the kernel.  LATEST_TOO, where more streams are listed, answers them by the latest positions
// in the same launch: as a launch before this one, which leaves at once where few are listed, it took those calls 6 us per layer.
enum ContextForm { PLAIN, IN_PARTS, LATEST_TOO };
template <int NT, bool TOGETHER, int FORM = PLAIN>
__global__ void __launch_bounds__(NT, NT > 512 ? 1 : NT > 256 ? 2 : 5)
rosa_context_kernel(const uint32_t* __restrict__ q_sw, const uint32_t* __restrict__ k_sw, const uint32_t* __restrict__ v_sw,
                    uint32_t* __restrict__ idx_sw, const uint32_t* __restrict__ list, const uint32_t* __restrict__ count,
                    uint32_t* __restrict__ next, uint32_t* __restrict__ hard, uint32_t* __restrict__ hard_count, uint32_t T,
                    size_t wps, uint32_t easy_bits, ContextLimits limits, uint32_t from, uint32_t to, HeadsCall heads_call) {
    chain_entry();
    constexpr uint32_t NW = NT / 32, BRUTE = context::BRUTE;
    extern __shared__ __align__(16) uint8_t context_mem[];
    __shared__ uint32_t sh_item, sh_sums[NW], sh_pairs[NW], sh_gone, sh_large;
    const uint32_t words = (T + 31u) / 32u, uneven_bits = TOGETHER ? context::bits_for_uneven(T) : easy_bits;
    const ContextLayout L(T, uneven_bits, NW);
    uint16_t* hist = reinterpret_cast<uint16_t*>(context_mem + L.hist);
    uint32_t* hist2 = reinterpret_cast<uint32_t*>(context_mem + L.hist);   // two counts per word
    uint16_t* start = reinterpret_cast<uint16_t*>(context_mem + L.start);
    uint32_t* start2 = reinterpret_cast<uint32_t*>(context_mem + L.start);
    uint32_t* Q = reinterpret_cast<uint32_t*>(context_mem + L.q);
    uint32_t* K = reinterpret_cast<uint32_t*>(context_mem + L.k);
    uint32_t* V = reinterpret_cast<uint32_t*>(context_mem + L.v);
    uint16_t* q_ends = reinterpret_cast<uint16_t*>(context_mem + L.q_ends);
    uint16_t* k_ends = reinterpret_cast<uint16_t*>(context_mem + L.k_ends);
    uint16_t* in_word = reinterpret_cast<uint16_t*>(context_mem + L.in_word);
    uint32_t* before_word = reinterpret_cast<uint32_t*>(context_mem + L.before);
    uint32_t* out_s = reinterpret_cast<uint32_t*>(context_mem + L.out);
    context::Entry* entries = reinterpret_cast<context::Entry*>(context_mem + L.entries);
    uint16_t* steps = reinterpret_cast<uint16_t*>(context_mem + L.steps);
    uint16_t* large_steps = hist;   // after the sort; NW * C > T entries for the 16 warps of TOGETHER
    const context::Runs runs{k_ends, in_word, before_word};
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t total = *count;
    const bool contexts_for_all = FORM == LATEST_TOO && *heads_call.uneven_count * UNEVEN_SHARE > total;   // 0 where they were not counted
    if (FORM == LATEST_TOO && total >= to && !contexts_for_all) {
        heads_streams(q_sw, k_sw, v_sw, idx_sw, list, total, T, wps, context_mem, heads_call);
        return;
    }
    if (total < from || (total >= to && !contexts_for_all)) return;
    const uint32_t parts = FORM == IN_PARTS && total ? min(max(gridDim.x / total, 1u), MAX_PARTS) : 1u;
    const uint32_t rows_per_warp = (words + NW - 1u) / NW;
    const uint32_t row0 = min(warp * rows_per_warp, words), row1 = min(row0 + rows_per_warp, words);   // a warp's keys
    for (;;) {
        __syncthreads();   // the stream before this one is done with everything below
        if (threadIdx.x == 0) {
            sh_item = atomicAdd(next, 1u);
            sh_gone = 0u;
            sh_large = 0u;
        }
        __syncthreads();
        if (sh_item >= total * parts) return;
        // Every parts-th row of 32 steps is this part's own: it sorts for itself, in an order of its own within a bucket.
        const uint32_t part = FORM == IN_PARTS ? sh_item / total : 0u;
        const auto own_row = [&](uint32_t row) { return parts == 1u || row % parts == part; };
        const size_t s = list[FORM == IN_PARTS ? sh_item % total : sh_item];
        for (uint32_t w = threadIdx.x; w < words; w += NT) {
            Q[w + 1u] = q_sw[s * wps + w];
            K[w + 1u] = k_sw[s * wps + w];
            if (TOGETHER) V[w] = v_sw[s * wps + w];
            out_s[w] = 0u;
        }
        if (threadIdx.x == 0) Q[0] = K[0] = 0u;
        bool by_runs = false, taken = false, sorted = false;   // sorted: the steps bucket by bucket too
        uint32_t c = easy_bits, C = 1u << c, pair_words = C / 2u;
        uint32_t* nq2 = hist2 + NW * pair_words;   // the same counts of the steps
        uint32_t pairs_by_bits = 0;
        auto key_of_key = [&](uint32_t r) {
            return by_runs ? context::run_key(K, k_ends, r, c) : context::window(K, r) >> (32u - c);
        };
        auto key_of_step = [&](uint32_t t) {
            return by_runs ? context::run_key(Q, q_ends, t, c) : context::window(Q, t) >> (32u - c);
        };
        for (int attempt = 0;; ++attempt) {
            if (TOGETHER && attempt == 1) {
                c = uneven_bits;
                C = 1u << c;
                pair_words = C / 2u;
                nq2 = hist2 + NW * pair_words;
            }
            for (uint32_t i = threadIdx.x; i < (NW + 1u) * pair_words; i += NT) hist2[i] = 0u;   // hist and nq
            __syncthreads();
            for (uint32_t row = row0; row < row1; ++row) {
                const uint32_t r = row * 32u + lane;
                if (r < T) {
                    const uint32_t ck = key_of_key(r);
                    atomicAdd(&hist2[warp * pair_words + (ck >> 1)], 1u << ((ck & 1u) * 16u));
                    if (r >= BRUTE && own_row(row)) {
                        const uint32_t cq = key_of_step(r);
                        atomicAdd(&nq2[cq >> 1], 1u << ((cq & 1u) * 16u));
                    }
                }
            }
            __syncthreads();
            // exclusive sums over the buckets (keys in the low half, steps in the high half), and the number of pairs
            const uint32_t per = (pair_words + NT - 1u) / NT;
            const uint32_t j0 = min(threadIdx.x * per, pair_words), j1 = min(j0 + per, pair_words);
            uint32_t sum = 0, pairs = 0;
            for (uint32_t j = j0; j < j1; ++j) {
                uint32_t n = 0;
#pragma unroll 8
                for (uint32_t w = 0; w < NW; ++w) n += hist2[w * pair_words + j];
                start2[j] = n;
                const uint32_t m = nq2[j];
                pairs += (n & 0xFFFFu) * (m & 0xFFFFu) + (n >> 16) * (m >> 16);
                sum += (n & 0xFFFFu) + (n >> 16) + (((m & 0xFFFFu) + (m >> 16)) << 16);
            }
            uint32_t before = sum;
#pragma unroll
            for (uint32_t o = 1; o < 32u; o <<= 1) {
                const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, before, o);
                if (lane >= o) before += x;
            }
            pairs = __reduce_add_sync(0xFFFFFFFFu, pairs);
            if (lane == 31u) {
                sh_sums[warp] = before;
                sh_pairs[warp] = pairs;
            }
            __syncthreads();
            uint32_t run = before - sum;
            pairs = 0;
            for (uint32_t w = 0; w < NW; ++w) {
                if (w < warp) run += sh_sums[w];
                pairs += sh_pairs[w];
            }
            pairs *= parts;   // about what all of them have
            // By bits when that is easy; otherwise by whichever of the two ways has fewer pairs, if those are few enough.
            if (attempt == 0) {
                taken = pairs <= limits.easy * T;
                pairs_by_bits = pairs;
            } else if (attempt == 1) {
                taken = pairs <= pairs_by_bits && pairs <= limits.by_runs * T;
            } else {
                taken = true;
            }
            if (taken) {
                // two buckets side by side, eight counts in flight (one after the other they were 64 trips for 32 warps)
                uint32_t run_k = run & 0xFFFFu, run_q = run >> 16;
                for (uint32_t j = j0; j < j1; ++j) {
                    const uint32_t n = start2[j], m = nq2[j];
                    uint32_t at = run_k | (run_k + (n & 0xFFFFu)) << 16;
                    start2[j] = at;
                    for (uint32_t w0 = 0; w0 < NW; w0 += 8u) {
                        uint32_t counts[8];
#pragma unroll
                        for (uint32_t u = 0; u < 8u; ++u) counts[u] = hist2[(w0 + u) * pair_words + j];
#pragma unroll
                        for (uint32_t u = 0; u < 8u; ++u) {
                            hist2[(w0 + u) * pair_words + j] = at;
                            at += counts[u];
                        }
                    }
                    nq2[j] = run_q | (run_q + (m & 0xFFFFu)) << 16;
                    run_k += (n & 0xFFFFu) + (n >> 16);
                    run_q += (m & 0xFFFFu) + (m >> 16);
                }
                if (threadIdx.x == 0) start[C] = (uint16_t)T;
            }
            sorted = attempt != 0;
            if (taken || (attempt == 1 && pairs_by_bits > limits.by_bits * T)) break;
            by_runs = attempt == 0;
            if (by_runs) {
                for (uint32_t w = threadIdx.x; w < words; w += NT) {
                    q_ends[w] = (uint16_t)context::run_at_end(Q, w);
                    k_ends[w] = (uint16_t)context::run_at_end(K, w);
                }
            }
        }
        const auto leave = [&] {   // to rosa_match_kernel, by the first part that does
            if (parts == 1u || atomicExch(&heads_call.given_up[s], 2u) != 2u) hard[atomicAdd(hard_count, 1u)] = (uint32_t)s;
        };
        if (!taken) {
            if (threadIdx.x == 0) leave();
            continue;
        }
        __syncthreads();
        // a warp's keys in order: equal contexts of 32 steps take consecutive places
        for (uint32_t row = row0; row < row1; ++row) {
            const uint32_t r = row * 32u + lane;
            const uint32_t ck = r < T ? key_of_key(r) : 0xFFFFFFFFu;
            const uint32_t same = __match_any_sync(0xFFFFFFFFu, ck);
            const uint32_t rank = __popc(same & ((1u << lane) - 1u));
            uint32_t at = 0;
            if (r < T) {
                at = hist[warp * C + ck];
                entries[at + rank] = context::Entry{context::window(K, r), r};
                if (sorted && r >= BRUTE && own_row(row)) {   // in any order within a bucket
                    const uint32_t cq = key_of_step(r), sh = (cq & 1u) * 16u;
                    steps[(atomicAdd(&nq2[cq >> 1], 1u << sh) >> sh) & 0xFFFFu] = (uint16_t)r;
                }
            }
            __syncwarp();
            if (r < T && rank == 0u) hist[warp * C + ck] = (uint16_t)(at + __popc(same));
            __syncwarp();
        }
        if (by_runs) {
            for (uint32_t i = threadIdx.x; i < 2u * words; i += NT) {
                const uint32_t b = i >= words, w = i - b * words;
                const uint32_t x = context::longest_in_word(K, k_ends, w, T, b);
                before_word[i] = x;
                in_word[i] = (uint16_t)(x >> 16);
            }
            __syncthreads();
            if (warp < 2u) {   // running maximum over the words, exclusive: a warp per bit
                uint32_t carry = 0;
                for (uint32_t w0 = 0; w0 < words; w0 += 32u) {
                    const uint32_t w = w0 + lane;
                    uint32_t x = w < words ? before_word[warp * words + w] : 0u;
#pragma unroll
                    for (uint32_t o = 1; o < 32u; o <<= 1) {
                        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                        if (lane >= o) x = max(x, y);
                    }
                    x = max(x, carry);
                    uint32_t excl = __shfl_up_sync(0xFFFFFFFFu, x, 1);
                    if (lane == 0) excl = carry;
                    __syncwarp();
                    if (w < words) before_word[warp * words + w] = excl;
                    carry = __shfl_sync(0xFFFFFFFFu, x, 31);
                }
            }
        }
        __syncthreads();
        // Easy streams step by step.  On the others the number of positions to look at differs a lot from bucket to bucket:
        // their steps are taken bucket by bucket, so that the lanes of a warp look through the same ones.
        // Many streams side by side hide the way to L1 and pay for the copy (four sequences 1.96 ms, with it 1.98); of few the slowest
        // stream is what lasts (one 0.88, with it 0.85).
        const uint32_t* v = TOGETHER ? V : v_sw + s * wps;
        uint32_t* out = idx_sw + s * wps;
        uint32_t deep = 0;
        const uint32_t most_deep = by_runs ? limits.deep_by_runs : limits.deep_by_bits;
        // Where a step's bucket lies, its best position within it (by the lanes of a warp where `together`: entries b + lane,
        // b + lane + 32, ...), and the answer.
        struct Step {
            uint32_t b, e, run;
            context::Query z;
        };
        auto find_bucket = [&](uint32_t t) {
            Step x;
            if (by_runs) {
                const uint32_t key = context::run_key(Q, q_ends, t, c);
                x.run = context::run_at(Q, q_ends, t);
                x.z.wq = context::window(Q, t);
                x.z.first = key;
                x.z.n = 1u;
            } else {
                x.run = 0u;
                x.z = context::query(Q, c, !sorted, t);
            }
            x.b = start[x.z.first];
            x.e = start[x.z.first + x.z.n];
            return x;
        };
        auto finish = [&](const Step& x, uint32_t t, uint32_t found, int32_t best) -> uint32_t {
            if (found) return found & 0xFFFFu;
            if (!by_runs) return context::find_shorter(entries, start, c, x.z, t, best);
            if (context::scan_agreement(best) > (int32_t)x.run) return context::scan_position(best) + 1u;
            return context::find_inside_run(K, runs, words, context::bit_at(Q, t), x.run, t, deep);
        };
        auto v_bit = [&](uint32_t r1) { return r1 ? (v[r1 >> 5] >> (r1 & 31u)) & 1u : 0u; };
        auto gone = [&] {   // by vote: lanes that read the flag apart from one another could disagree, and part for good
            if (!__any_sync(0xFFFFFFFFu, deep > most_deep || *static_cast<volatile uint32_t*>(&sh_gone) != 0u)) return false;
            if (lane == 0) sh_gone = 1u;
            return true;
        };
        if (TOGETHER) {   // the steps below BRUTE by a warp each
            for (uint32_t t = warp; t < min(BRUTE, T); t += NW) {
                if (!own_row(t >> 5)) continue;
                const uint32_t wq = context::window(Q, t);
                uint32_t best = 0;
                for (uint32_t r = lane; r < t; r += 32u) {
                    const uint32_t n = context::agreement(Q, K, t, r, wq ^ context::window(K, r), deep);
                    if (n) best = max(best, n << 16 | (r + 1u));
                }
                best = __reduce_max_sync(0xFFFFFFFFu, best);
                if (lane == 0 && v_bit(best & 0xFFFFu)) atomicOr(&out_s[t >> 5], 1u << (t & 31u));
            }
        }
        // The last rows first: they have the most keys to agree with, so a stream that has to be given up is at once.
        const uint32_t first_row = min(TOGETHER ? BRUTE / 32u : 0u, words);
        // The rows of this part (each may sort or not, by its own count of pairs), the sorted steps of which are in `steps`.
        const int32_t last_own = (int32_t)(words - 1u) - (int32_t)((words - 1u + parts - part) % parts);
        uint32_t n_rows = last_own >= (int32_t)first_row ? ((uint32_t)last_own - first_row) / parts + 1u : 0u, own_steps = 0;
        if (sorted) {
            if (last_own >= (int32_t)(BRUTE / 32u)) {
                own_steps = (((uint32_t)last_own - BRUTE / 32u) / parts + 1u) * 32u;
                if ((uint32_t)last_own == words - 1u) own_steps -= 32u * words - T;
            }
            n_rows = min(BRUTE / 32u, words) - first_row + (own_steps + 31u) / 32u;
        }
        for (uint32_t j = warp; j < n_rows; j += NW) {
            const uint32_t row = sorted ? first_row + j : (uint32_t)last_own - j * parts;
            const uint32_t i = row * 32u + lane, t = !sorted || i < BRUTE ? i : i - BRUTE < own_steps ? steps[i - BRUTE] : T;
            uint32_t r1 = 0;
            bool large = false;
            if (row * 32u < BRUTE) {
                if (t < T) r1 = context::find_brute(Q, K, t, deep);
            } else if (t < T) {
                const Step x = find_bucket(t);
                large = TOGETHER && (x.e - x.b) * t > CONTEXT_LARGE * T;   // about so many of them lie before t
                if (!large) {
                    uint32_t found = 0;
                    int32_t best = context::SCAN_NOTHING;
                    if (by_runs && x.run >= 32u) {
                        found = context::scan_runs(entries, x.b, x.e, 1u, Q, K, runs, x.run, t, deep);
                    } else {
                        best = context::scan(entries, start, x.z.first, x.z.n, t, x.z.wq, best);
                        if (context::scan_full(best)) found = context::scan_deep(entries, x.b, x.e, 1u, Q, K, x.z.wq, t, deep, most_deep);
                    }
                    r1 = finish(x, t, found, best);
                }
            }
            const uint32_t bit = v_bit(r1);
            if (sorted || TOGETHER) {
                if (bit) atomicOr(&out_s[t >> 5], 1u << (t & 31u));
            } else {
                const uint32_t word = __ballot_sync(0xFFFFFFFFu, bit != 0u);
                if (lane == 0) out[row] = word;
            }
            if (TOGETHER) {
                const uint32_t these = __ballot_sync(0xFFFFFFFFu, large);
                uint32_t at = 0;
                if (these && lane == 0) at = atomicAdd(&sh_large, (uint32_t)__popc(these));
                at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(these & ((1u << lane) - 1u));
                if (large) large_steps[at] = (uint16_t)t;
            }
            if (gone()) break;
        }
        if (TOGETHER) {
            // Large buckets a step per warp.  They lie side by side, so without this list they fell to a few warps (one
            // sequence of the default model: a row of 32 such steps took 100 000 cycles, the whole stream 300 000).
            __syncthreads();
            const uint32_t n_large = sh_large;
            for (uint32_t j = warp; j < n_large; j += NW) {
                const uint32_t t = large_steps[j];
                const Step x = find_bucket(t);
                uint32_t found = 0;
                int32_t best = context::SCAN_NOTHING;
                if (by_runs && x.run >= 32u) {
                    found = __reduce_max_sync(0xFFFFFFFFu, context::scan_runs(entries, x.b + lane, x.e, 32u, Q, K, runs, x.run, t, deep));
                } else {
                    for (uint32_t k = x.b + lane; k < x.e; k += 32u) best = context::scan_one(entries[k], t, x.z.wq, best);
                    best = __reduce_min_sync(0xFFFFFFFFu, best);
                    if (context::scan_full(best))
                        found = __reduce_max_sync(0xFFFFFFFFu, context::scan_deep(entries, x.b + lane, x.e, 32u, Q, K, x.z.wq, t, deep, most_deep));
                }
                const uint32_t bit = v_bit(finish(x, t, found, best));
                if (lane == 0 && bit) atomicOr(&out_s[t >> 5], 1u << (t & 31u));
                if (gone()) break;
            }
        }
        __syncthreads();
        if (sh_gone) {
            if (threadIdx.x == 0) leave();
        } else if (sorted || TOGETHER) {
            for (uint32_t w = threadIdx.x; w < words; w += NT)
                if (own_row(w)) out[w] = out_s[w];
        }
    }
}

// The remaining streams by sets of lags (rosa_match.cuh).  A work item is a piece of one stream, a warp takes items
// from a counter until they run out; the warps of a CTA have nothing to do with one another.
constexpr int MATCH_WARPS = 4;
constexpr uint32_t MATCH_COUNTS = 8;   // of MatchCall

// A stream whose query bits are all c: idx follows the longest run of c among the keys so far, the latest of equals
// (sam_core.cuh run_constant_q), a running maximum over (run length, position).  A lane has a word: the run that comes in from the words
// before follows from the full ones among them, the longest run so far from a scan over the words' maxima, and the v bit that a
// run leads to lies in the word or the one after it.  T <= 8192.  (With a lane per step and a scan per word, 64 words one after the other:
// one sequence of the default model, 2048 steps, 18 us a layer for this kernel, now 13.5; an empty launch between events takes 6.)
__device__ __forceinline__ void constant_q_warp(uint32_t c, const uint32_t* __restrict__ k, const uint32_t* __restrict__ v,
                                                uint32_t* __restrict__ out, uint32_t T) {
    constexpr uint32_t ALL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u, words = (T + 31u) / 32u;
    uint32_t run_before = 0, best = 0;   // run length << 15 | (position + 1) << 1 | v bit of the step after the position
    for (uint32_t w0 = 0; w0 < words; w0 += 32u) {
        const uint32_t w = w0 + lane, key = w < words ? k[w] : 0u, same = w < words ? c ? key : ~key : 0u;
        const uint32_t after = __funnelshift_r(w < words ? v[w] : 0u, w + 1u < words ? v[w + 1u] : 0u, 1u);   // bit b: v of step b + 1
        const uint32_t full = __ballot_sync(ALL, same == ALL), upper = (uint32_t)__clz((int)~same);
        const uint32_t z = lane ? min((uint32_t)__clz((int)~(full << (32u - lane))), lane) : 0u;   // full words right below
        const uint32_t there = __shfl_sync(ALL, upper, (int)(z < lane ? lane - 1u - z : 0u));
        const uint32_t run0 = 32u * z + (z < lane ? there : run_before);
        // the longest run that ends at a position of the word from `cur` on; bit b of the answer: what is known before position b
        const auto walk = [&](uint32_t cur, uint32_t& answer) {
            uint32_t run = run0;
#pragma unroll
            for (uint32_t b = 0; b < 32u; ++b) {
                answer |= (cur & 1u) << b;
                const bool is = same >> b & 1u;
                run = is ? run + 1u : 0u;
                const uint32_t x = run << 15 | (32u * w + b + 1u) << 1 | (after >> b & 1u);
                cur = is && x > cur ? x : cur;
            }
            return cur;
        };
        uint32_t unused = 0, word = 0, longest = walk(0u, unused);
#pragma unroll
        for (uint32_t o = 1; o < 32u; o <<= 1) {
            const uint32_t x = __shfl_up_sync(ALL, longest, o);
            if (lane >= o) longest = max(longest, x);
        }
        const uint32_t below = __shfl_up_sync(ALL, longest, 1);
        walk(lane ? max(best, below) : best, word);
        if (w + 1u == words && (T & 31u)) word &= (1u << (T & 31u)) - 1u;
        if (w < words) out[w] = word;
        best = max(best, __shfl_sync(ALL, longest, 31));
        run_before = __shfl_sync(ALL, same == ALL ? run0 + 32u : upper, 31);
    }
}

template <int NW>
__global__ void __launch_bounds__(32 * MATCH_WARPS)
rosa_match_kernel(const uint32_t* __restrict__ q_sw, const uint32_t* __restrict__ k_sw, const uint32_t* __restrict__ v_sw,
                  uint32_t* __restrict__ idx_sw, const uint32_t* __restrict__ hard, const uint32_t* __restrict__ hard_count,
                  const uint32_t* __restrict__ cq_list, const uint32_t* __restrict__ cq_count, uint32_t* __restrict__ next,
                  uint32_t* __restrict__ clear, uint32_t* __restrict__ kept, uint32_t T, size_t wps, uint32_t ring_words) {
    chain_entry();
    if (blockIdx.x == 0 && threadIdx.x < MATCH_COUNTS) clear[threadIdx.x] = 0u;   // the counters of the next call
    extern __shared__ __align__(16) uint32_t match_mem[];
    const match::Layout L(NW, ring_words);
    uint32_t* mem = match_mem + (threadIdx.x >> 5) * L.total;
    kept += (size_t)(blockIdx.x * MATCH_WARPS + (threadIdx.x >> 5)) * (match::CHECKPOINTS * 32u * NW);
    const uint32_t gap = match::checkpoint_gap(T);
    const uint32_t total = *hard_count, constant = *cq_count;
    // Pieces as long as the number of streams allows: a piece costs its set-up and the search for its first window
    // on top of its steps, but the device wants a few pieces per warp.
    const uint32_t warps = gridDim.x * MATCH_WARPS;
    uint32_t piece = 1024u * NW;
    while (piece > 32u && (uint64_t)total * ((T + piece - 1u) / piece) < 3ull * warps) piece >>= 1;
    const uint32_t pieces = (T + piece - 1u) / piece;
    const uint32_t items = total * pieces;   // below 2^32: the host checked it for the shortest pieces
    // The first item of a warp is its own number, so that the many without one leave without a word to anybody.
    for (uint32_t item = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; item < items + constant;
         item = warps + __shfl_sync(0xFFFFFFFFu, (threadIdx.x & 31u) == 0u ? atomicAdd(next, 1u) : 0u, 0)) {
        if (item >= items) {
            const size_t s = cq_list[item - items];
            constant_q_warp(q_sw[s * wps] & 1u, k_sw + s * wps, v_sw + s * wps, idx_sw + s * wps, T);
            continue;
        }
        const uint32_t i = item % total, t0 = (pieces - 1u - item / total) * piece, t1 = min(t0 + piece, T);   // the wide sets first
        const size_t s = hard[i];
        const uint32_t *q = q_sw + s * wps, *k = k_sw + s * wps, *v = v_sw + s * wps;
        uint32_t* out = idx_sw + s * wps;
        if (NW >= 8 && t1 > 4096u) match::piece<8>(mem, L, ring_words, kept, gap, q, k, v, out, t0, t1);
        else if (NW >= 4 && t1 > 2048u) match::piece<4>(mem, L, ring_words, kept, gap, q, k, v, out, t0, t1);
        else if (NW >= 2 && t1 > 1024u) match::piece<2>(mem, L, ring_words, kept, gap, q, k, v, out, t0, t1);
        else match::piece<1>(mem, L, ring_words, kept, gap, q, k, v, out, t0, t1);
    }
}

constexpr uint32_t LEFT_PER_SM = 6;   // streams, beyond which they are many (`contexts`)
constexpr size_t MATCH_MAX_TIME = 8192;   // 256 words of lags, eight per lane
constexpr uint32_t HEADS_MAX_TIME = 2048;
constexpr size_t SM_SMEM = 228 * 1024, CTA_SMEM = 1536;   // of an SM; what a CTA needs beside its dynamic part, reserved and static

struct MatchCall {   // the buffers of one call
    const uint32_t *q, *k, *v;
    uint32_t *idx, *list, *cq_list, *hard, *left, *given_up;
    // listed, constant q, hard, next of the contexts, next of the matches, left by the latest positions, their next, listed and uneven; those
    // of the next call
    uint32_t *counts, *clear;
    size_t streams, wps;
    uint32_t T;
    ContextForm form;
};

// The shapes of the context kernel: threads per stream, and whether a warp takes a large bucket together.
enum ContextShape { CONTEXT_256, CONTEXT_512, CONTEXT_1024, CONTEXT_SHAPES };

template <int NT, bool TOGETHER>
void prepare_context(ullis_cuda_runtime* rt, uint32_t T, int shape) {
    const auto kernel = rosa_context_kernel<NT, TOGETHER>;
    const size_t smem = ContextLayout(T, context_bits(T, TOGETHER), NT / 32).total;
    if (!rt->context_smem[shape]) {   // the attribute belongs to the function, not to this runtime: always the same value
        const size_t most = ContextLayout((uint32_t)MATCH_MAX_TIME, context::bits_for((uint32_t)MATCH_MAX_TIME), NT / 32).total;
        ULLIS_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
        if constexpr (TOGETHER)
            ULLIS_CUDA_CHECK(cudaFuncSetAttribute(rosa_context_kernel<NT, TOGETHER, IN_PARTS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
        ULLIS_CUDA_CHECK(cudaFuncSetAttribute(rosa_context_kernel<NT, TOGETHER, LATEST_TOO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(SM_SMEM - CTA_SMEM)));
    }
    if (rt->context_smem[shape] != smem) {
        int per_sm = 0;
        ULLIS_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, NT, smem));
        rt->context_ctas[shape] = std::max(1, per_sm) * rt->sm_count;
        rt->context_smem[shape] = smem;
    }
}

template <int NT, bool TOGETHER>
void launch_context(ullis_cuda_runtime* rt, const MatchCall& m, int shape, ContextForm form, const uint32_t* list, const uint32_t* count, uint32_t from,
                    uint32_t to, const char* what) {
    const unsigned grid = (unsigned)std::min<size_t>(rt->context_ctas[shape], m.streams);
    // A match kernel step costs about as much as 100 positions here; up to 24 the lanes are even enough without sorting
    // the steps.  What a thread has compared when its stream turns out to repeat itself is thrown away: by bits 64 long
    // comparisons tell (streams of clean periods 16 to 256, 2048 steps, 512 / 8192 of them: contexts 0.37 / 2.12 ms with
    // 256, now 0.13 / 0.67), by runs 256 (with 64, 64 sequences of the default model 33.3 ms, not 29.8: streams that hardly
    // ever change went to the match kernel).
    const ContextLimits limits{24u, 96u, 160u, 64u, 256u};
    size_t smem = rt->context_smem[shape];
    HeadsCall heads{0u, 1u, 128u, 40u, m.counts + 6, m.left, m.counts + 5, m.given_up, m.counts + 7};
    auto kernel = rosa_context_kernel<NT, TOGETHER>;
    if (form == LATEST_TOO) {
        kernel = rosa_context_kernel<NT, TOGETHER, LATEST_TOO>;
        // As many warps as have room beside each other with the CTAs that an SM holds anyway (2048 steps: 23 with 1024 threads, 22 with 512, 20
        // with 256).
        const size_t per_sm = (size_t)rt->context_ctas[shape] / rt->sm_count, each = HeadsLayout(m.T).total;
        heads.warps = (uint32_t)std::min<size_t>(NT / 32, (SM_SMEM / per_sm - CTA_SMEM) / each);
        smem = std::max(smem, heads.warps * each);
        // More pieces make a launch of few streams shorter and one of many longer, since their warps put in the same keys again.  Below
        // 1024 steps a piece costs more than it saves unless warps would be idle (gain 1 + N(0, 0.02), ROSA kernels in all layers with 20
        // warps per SM, 1 / 2 / 4 pieces: 16 times 700 steps of the default model 1.51 / 1.66 / 1.81 ms, 3 times 333 of the small one 0.255 /
        // 0.235 / 0.236; 2048 steps of the default model: 4 sequences 2.90 / 2.45 / 2.10, 8 3.71 / 3.11 / 2.99, 16 5.09 / 4.75 / 4.97, 64 14.0 /
        // 14.4 / 16.7).
        const size_t warps = (size_t)rt->context_ctas[shape] * heads.warps;
        const uint32_t wanted = m.T < 1024u ? (m.streams * 4u <= warps ? 4u : 1u) : m.streams * 2u < 3u * warps ? 4u : m.streams < 8u * warps ? 2u : 1u;
        heads.pieces = heads::pieces_with_rows((m.T + 31u) / 32u, wanted);
        // heads.base, heads.per_row: less leaves the contexts streams that are cheaper here (whole calls with 12 / 16 / 24 / 40 per row, ms:
        // 16 times 2048 steps 9.70 / 9.61 / 9.57 / 9.46, 16 times 1100 5.37 / 5.35 / 5.25 / 5.13, 5 times 1531 3.38 / 3.36 / 3.36 / 3.31), and a base
        // too small all that are short (ROSA kernels of twice 700 steps, base 32 / 64 / 128: 0.75 / 0.62 / 0.61).
    } else if constexpr (TOGETHER) {
        if (form == IN_PARTS) kernel = rosa_context_kernel<NT, TOGETHER, IN_PARTS>;
    }
    rt->chain(kernel, grid, NT, smem, m.q, m.k, m.v, m.idx, list, count, m.counts + 3, m.hard, m.counts + 2, m.T, m.wps, context::bits_for(m.T), limits,
              from, to, heads);
    rt->launched(what);
}

template <int NW>
void launch_match(ullis_cuda_runtime* rt, const MatchCall& m, int slot, uint32_t ring_words) {
    const match::Layout L(NW, ring_words);
    const size_t smem = (size_t)L.total * 4u * MATCH_WARPS;
    if (!rt->match_ctas[slot]) {
        int per_sm = 0;
        ULLIS_CUDA_CHECK(cudaFuncSetAttribute(rosa_match_kernel<NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        ULLIS_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, rosa_match_kernel<NW>, 32 * MATCH_WARPS, smem));
        rt->match_ctas[slot] = std::max(1, per_sm) * rt->sm_count;
    }
    const size_t most = (m.streams * m.wps + MATCH_WARPS - 1) / MATCH_WARPS;   // every stream in the shortest pieces
    // the kept sets count against the same cap on scratch memory as the automaton's states (32 KB * NW per CTA)
    const size_t kept_words = (size_t)MATCH_WARPS * match::CHECKPOINTS * 32u * NW;
    const size_t allowed = std::max<size_t>(1, rt->sam_budget_bytes / (kept_words * 4));
    const unsigned grid = (unsigned)std::min({(size_t)rt->match_ctas[slot], most, allowed});
    uint32_t* kept = rt->sam_scratch.as<uint32_t>((size_t)grid * kept_words);
    rt->chain(rosa_match_kernel<NW>, grid, 32 * MATCH_WARPS, smem, m.q, m.k, m.v, m.idx, m.hard, m.counts + 2,
              m.cq_list, m.counts + 1, m.counts + 4, m.clear, kept, m.T, m.wps, ring_words);
    rt->launched("rosa_match");
}

// EAGER keeps the reference's schedule for every stream (no shortcut): list = all streams
__global__ void rosa_list_all_kernel(uint32_t* __restrict__ list, uint32_t* __restrict__ count, size_t streams) {
    const size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s < streams) list[s] = (uint32_t)s;
    if (s == 0) *count = (uint32_t)streams;
}

template <typename Ix>
size_t stride_for(int algo, size_t T) {
    return algo == ULLIS_CUDA_SAM_EAGER ? sam::EagerLayout<Ix>((uint32_t)T).total
                                        : sam::EulerLayout<Ix>((uint32_t)T).total;
}

// The listed streams by the latest positions or by contexts, in the shapes that suit how many there are.  That number is known on the device only,
// where a launch whose range it misses leaves at once: one launch for the calls where most streams had a closed form, whose
// others are uneven (large buckets), one for the rest - a single one where both are of the same shape.
//
// Many streams: the shape with the most warps per SM, which shared memory decides - up to T = 4096 256 threads, for 8192
// steps (110 KB of shared memory at 256 threads, 160 at 1024) 1024.  Fewer streams than SMs: a launch lasts as long as one
// stream, so 1024 threads.  Between them larger blocks pay the more the fewer and the more uneven the streams are.  Context
// kernels in us, 256 / 512 / 1024 threads, all streams listed, i.i.d. bits and bits of probabilities 0.002 to 0.99:
//
//     streams         96 *                512                    1024                     4096           (* T = 6000: 128)
//     T = 300     15 / 13 / 14         16 / 20 / 33           27 / 33 / 53            67 / 98 / 186
//                 26 / 29 / 29         31 / 35 / 47           38 / 49 / 74            82 / 127 / 231
//     T = 700     18 / 16 / 16         21 / 29 / 37           33 / 47 / 62            89 / 145 / 221
//                 61 / 39 / 33         57 / 53 / 61           88 / 86 / 106          193 / 234 / 334
//     T = 2048    33 / 27 / 25         46 / 51 / 66           74 / 90 / 121          205 / 291 / 414
//                158 / 119 / 76       205 / 154 / 145        268 / 225 / 225         596 / 686 / 788
//     T = 6000    90 / 72 / 61        158 / 123 / 139        229 / 219 / 256         698 / 715 / 907
//                586 / 512 / 293      811 / 592 / 430        895 / 766 / 643        2080 / 1972 / 1997
//     T = 8192   109 / 80 / 68        248 / 250 / 201        414 / 453 / 363        1352 / 1649 / 1337
//                670 / 487 / 375     1077 / 745 / 573       1147 / 1120 / 754       3067 / 3227 / 2364
//
// Most streams listed: 512 threads up to 6 streams per SM (layers of the default model with gain 1 + N(0, 0.02), 2048 steps:
// one sequence 0.89 / 0.80 ms in all layers, two 1.22 / 1.31, three 1.54 / 1.81); below 1024 steps up to 7, where one launch then
// takes both kinds (small model, gain N(0, 0.02), 4 times 512 steps 0.17 ms, with a launch for each 0.20).
// Few listed: 1024 threads the longer the more streams there are.  One stream in eight listed, the others constant, 512 / 1024
// threads: T = 1024, 2048 streams 47 / 49, 4096 68 / 70, 8192 100 / 121; T = 1531, 4096 112 / 109, 6144 129 / 144; T = 2048,
// 4096 152 / 137, 6144 199 / 190, 8192 233 / 238; T = 4096, 8192 539 / 451.  Layers of the default model with gain N(0, 0.02),
// 2048 steps: one sequence 1.20 / 0.79 ms, 4 1.41 / 1.00, 8 1.63 / 1.48, 12 1.99 / 1.96, 16 2.33 / 2.43, 64 6.94 / 8.31.
//
// (Where the latest positions take the calls with most streams listed - context_form - the columns of so many streams are those of what
// they leave.)
void contexts(ullis_cuda_runtime* rt, const MatchCall& m) {
    prepare_context<256, false>(rt, m.T, CONTEXT_256);
    prepare_context<512, true>(rt, m.T, CONTEXT_512);
    prepare_context<1024, true>(rt, m.T, CONTEXT_1024);
    const size_t sms = (size_t)rt->sm_count;
    int many = CONTEXT_256;
    for (int shape = CONTEXT_512; shape < CONTEXT_SHAPES; ++shape)
        if (rt->context_ctas[shape] << shape > rt->context_ctas[many] << many) many = shape;
    int uneven, rest;
    if (m.T < 512u) {   // too few steps for many warps
        uneven = rest = m.streams <= (size_t)rt->context_ctas[CONTEXT_512] ? (int)CONTEXT_512 : many;
    } else if (m.streams <= sms) {
        uneven = rest = CONTEXT_1024;
    } else if (m.T < 1024u && m.streams > 56u * sms) {   // 64 times 300 steps of the default model 4.7 ms with 256 threads alone, 5.1
        uneven = rest = many;
    } else {
        uneven = std::max<int>(many, m.T >= 1024u && m.streams * 50u <= m.T * sms ? CONTEXT_1024 : CONTEXT_512);
        rest = std::max<int>(many, m.streams <= (m.T < 1024u ? 7u : 6u) * sms ? CONTEXT_512 : CONTEXT_256);
    }
    const uint32_t all = ~0u, half = uneven == rest && m.form != LATEST_TOO ? all : (uint32_t)(m.streams / 2) + 1u;
    auto launch = [&](int shape, ContextForm form, const uint32_t* list, const uint32_t* count, uint32_t from, uint32_t to, const char* what) {
        if (shape == CONTEXT_256) launch_context<256, false>(rt, m, shape, form, list, count, from, to, what);
        else if (shape == CONTEXT_512) launch_context<512, true>(rt, m, shape, form, list, count, from, to, what);
        else launch_context<1024, true>(rt, m, shape, form, list, count, from, to, what);
    };
    if (m.form == LATEST_TOO) {
        // What the latest positions leave: few streams in parts, many of them in the shape of many, from where `rest` has that one.  In one launch,
        // in parts, many took twice the time (all of 2560 streams of 2048 steps left, bits of probability 0.9 1208 / 704 us, of clean periods
        // 928 / 254, 8192 of them 3281 / 2093 and 1315 / 670); a launch that leaves at once costs 1.5 us a layer.
        const uint32_t many_left = rest == uneven ? all : LEFT_PER_SM * (uint32_t)sms + 1u;
        launch(uneven, m.form, m.list, m.counts, 0u, half, "rosa_context");
        launch(uneven, IN_PARTS, m.left, m.counts + 5, 1u, many_left, "rosa_context_left");
        if (many_left != all) launch(rest, PLAIN, m.left, m.counts + 5, many_left, all, "rosa_context_left_many");
        return;
    }
    launch(uneven, m.form, m.list, m.counts, 0u, half, "rosa_context");
    if (half != all) launch(rest, PLAIN, m.list, m.counts, half, all, "rosa_context_even");
}

// How the listed streams of a call are to be answered.
ContextForm context_form(const ullis_cuda_runtime* rt, size_t streams, uint32_t T) {
    const size_t sms = (size_t)rt->sm_count;
    // The latest positions, where most streams are listed: one warp per stream or piece, so there have to be enough of them (all layers,
    // gain 1 + N(0, 0.02), contexts / latest positions, ms; 2048 steps: two sequences of the default model 1.57 / 1.73, three 1.83 / 1.93, four
    // 2.18 / 2.05, eight 3.49 / 2.82, 64 21.7 / 13.1; 1100 steps: two 1.01 / 1.06, four 1.39 / 1.25; 700: one 0.58 / 0.69, two 0.81 / 0.62, 16 2.57 / 1.49;
    // 300: two 0.51 / 0.45, 64 5.88 / 1.98).  Where few are listed those are uneven, and their chains long: 64 times 2048 steps with gain
    // N(0, 0.02) 7.7 / 9.3.  How uneven the listed ones are is not known here: a call of nothing but uneven streams takes 1 to 1.2 times as long as by
    // contexts alone, 5 x 2048 of clean periods 608 / 496 us, at worst 1.5 times (4 x 700 of all probabilities 209 / 141).  Beyond 2048 steps chains and tables grow (8192 steps of bits of probability 0.25 to 0.6: 1.09 / 1.63).
    if (T <= HEADS_MAX_TIME && streams > (T < 512u ? 4u : T < 1024u ? 5u : 14u) * sms) return LATEST_TOO;
    // Only a call of few streams can list less than half as many as there are CTAs.
    return streams <= PARTS_MAX_STREAMS * sms ? IN_PARTS : PLAIN;
}

// The whole call without an automaton: classification, the listed streams by contexts, and by sets of lags those that
// the contexts leave and the ones with a constant q.
void rosa_match(ullis_cuda_runtime* rt, const uint32_t* q_sw, const uint32_t* k_sw, const uint32_t* v_sw, uint32_t* idx_sw,
                size_t streams, uint32_t T) {
    MatchCall m;
    m.q = q_sw; m.k = k_sw; m.v = v_sw; m.idx = idx_sw;
    m.streams = streams; m.T = T; m.wps = (T + 31u) / 32u;
    m.list = rt->sam_list.as<uint32_t>(5 * streams);
    m.cq_list = m.list + streams;
    m.hard = m.cq_list + streams;
    m.left = m.hard + streams;
    m.given_up = m.left + streams;
    m.form = context_form(rt, streams, T);
    rt->counters(rt->match_counters, MATCH_COUNTS, &m.counts, &m.clear);
    rt->sam_last_counts = m.counts;
    rt->sam_last_streams = streams;
    if (!rt->parent) rt->lanes_last = 1;
    // Few short streams by the latest positions last as long as the longest walk, and what is given up as long again.  If more than one listed
    // stream in UNEVEN_SHARE is uneven all are answered by contexts.  us of the ROSA kernels, without / with the count: 4 x 300 x 512 bits of
    // probability 0.9 121 / 84, of slow changes 139 / 82, one half of those 120 / 74, even ones 39 / 41; 4 x 128 72 / 63, 86 / 68, 78 / 63, 31 / 32; 4 x 500 211 /
    // 133, 199 / 119, 160 / 95, 45 / 47; 8 x 400 238 / 177, 239 / 158, 173 / 127, 53 / 53.  Not at 16 x 600 (522 / 570, 456 / 449, 268 / 355), nor at 8 x 64 (43 / 73,
    // 45 / 70, 43 / 73).  No model in training has so many of them.
    const bool count_uneven = m.form == LATEST_TOO && T >= 128u && T < 512u && streams <= 28u * (size_t)rt->sm_count;
    rt->chain(count_uneven ? rosa_classify_kernel<true> : rosa_classify_kernel<false>, (unsigned)((streams * CLASSIFY_LANES + 127) / 128), 128, 0, q_sw, k_sw,
              v_sw, idx_sw, streams, T, m.wps, m.list, m.counts, m.cq_list, m.counts + 1, m.given_up, m.counts + 7);
    rt->launched("rosa_classify");
    contexts(rt, m);
    if (T <= 1024u) launch_match<1>(rt, m, 0, 1024);
    else if (T <= 2048u) launch_match<2>(rt, m, 1, 1024);
    else if (T <= 4096u) launch_match<4>(rt, m, 2, 2048);
    else launch_match<8>(rt, m, 3, 4096);
    rt->counters_cleared(rt->match_counters);
}

}  // namespace

size_t rosa_sam_scratch_bytes_per_stream(int algo, size_t time) {
    const bool narrow = sam::node_capacity((uint32_t)time) <= 0xFFFFu;
    return narrow ? stride_for<uint16_t>(algo, time) : stride_for<uint32_t>(algo, time);
}

bool rosa_without_automaton(const ullis_cuda_runtime* rt, size_t streams, size_t time) {
    return rt->sam_algo == ULLIS_CUDA_SAM_EULER && !rt->sam_automaton && time <= MATCH_MAX_TIME && streams * ((time + 31) / 32) < 0x7FFFFFFFull;
}

void rosa_sam(ullis_cuda_runtime* rt, const uint32_t* q_sw, const uint32_t* k_sw, const uint32_t* v_sw,
              uint32_t* idx_sw, size_t streams, size_t time, int site) {
    if (streams == 0 || time == 0) return;
    if (time > 0x3FFFFFFFu) fail(ULLIS_CUDA_ERR_SHAPE, "ROSA time does not fit 32-bit state ids");
    const int algo = rt->sam_algo;
    if (streams > 0xFFFFFFFFull) fail(ULLIS_CUDA_ERR_SHAPE, "too many ROSA streams");
    rt->sam_shares = 1;
    if (rosa_without_automaton(rt, streams, time)) {
        rosa_match(rt, q_sw, k_sw, v_sw, idx_sw, streams, (uint32_t)time);
        return;
    }
    const bool narrow = sam::node_capacity((uint32_t)time) <= 0xFFFFu;
    const size_t stride = rosa_sam_scratch_bytes_per_stream(algo, time);
    const size_t wps = (time + 31) / 32;
    // wave size: all streams at once when the scratch buffer already holds them;
    // otherwise bounded scratch (12 GiB unless ULLIS_CUDA_SAM_BUDGET_MB says otherwise, or what fits in free memory).
    // The memory query is a blocking driver call, so it is kept off the steady state.
    size_t wave = streams;
    if (rt->sam_scratch.bytes() < streams * stride) {
        size_t free_b = 0, total_b = 0;
        ULLIS_CUDA_CHECK(cudaMemGetInfo(&free_b, &total_b));
        size_t budget = rt->sam_budget_bytes;
        const size_t avail = free_b + rt->sam_scratch.bytes();  // what the scratch buffer could grow to
        if (avail < budget + ((size_t)2 << 30)) budget = avail > ((size_t)4 << 30) ? avail - ((size_t)2 << 30) : avail / 2;
        wave = budget / stride;
        if (wave == 0) fail(ULLIS_CUDA_ERR_NOMEM, "not enough device memory for one suffix-automaton state block");
        if (wave > streams) wave = streams;
    }
    uint8_t* scratch = static_cast<uint8_t*>(rt->sam_scratch.ensure(wave * stride));
    uint32_t* list = rt->sam_list.as<uint32_t>(2 * streams + 3);
    rt->sam_last_streams = streams;
    if (!rt->parent) rt->lanes_last = 1;   // a forward that splits its batch raises this after its last layer
    uint32_t* count = list + streams;
    rt->sam_last_counts = count;
    uint32_t* cq_count = count + 1;           // the constant-q streams, settled by a kernel of their own
    uint32_t* cq_list = count + 3;
    const unsigned cgrid = (unsigned)((streams + 127) / 128);
    // The number of streams left for the automaton is only known on the device;
    // each wave is sized for the worst case and surplus threads exit at once.
    const sam::CoopLayout coop((uint32_t)time);
    const bool use_coop = algo == ULLIS_CUDA_SAM_EULER && narrow && rt->sam_coop && coop.total <= 226 * 1024 &&
                          2 * sam::node_capacity((uint32_t)time) < 0xFFFFu;
    // The constant-q kernel runs on the side stream from the fork below until `stream` has waited for side_join.
    // Whichever way this function leaves in between (a launch error throws), the wait is issued: the next call
    // clears the counters and lists that kernel still reads.
    struct SideJoin {
        ullis_cuda_runtime* rt;
        bool forked = false;
        ~SideJoin() {
            if (forked) cudaStreamWaitEvent(rt->stream, rt->side_join, 0);
        }
    } side{rt};
    if (algo == ULLIS_CUDA_SAM_EAGER) {
        rosa_list_all_kernel<<<cgrid, 128, 0, rt->stream>>>(list, count, streams);
        rt->launched("rosa_list_all");
    } else {
        rt->zero(count, 8);   // both counters
        const unsigned classify_grid = (unsigned)((streams * CLASSIFY_LANES + 127) / 128);
        rt->chain(rosa_classify_kernel<false>, classify_grid, 128, 0, q_sw, k_sw, v_sw, idx_sw, streams, (uint32_t)time, wps, list,
                                                             count, cq_list, cq_count, nullptr, nullptr);
        rt->launched("rosa_classify");
        // The constant-q scan is a long serial loop for a few thousand threads; it depends on nothing but the
        // classification and writes idx words no other kernel of this call touches, so it runs on the side stream
        // beside the automaton pass (which is bound by latency and leaves most issue slots free).
        if (rt->sam_side) {
            if (!rt->side_stream) {
                ULLIS_CUDA_CHECK(cudaStreamCreateWithFlags(&rt->side_stream, cudaStreamNonBlocking));
                ULLIS_CUDA_CHECK(cudaEventCreateWithFlags(&rt->side_fork, cudaEventDisableTiming));
                ULLIS_CUDA_CHECK(cudaEventCreateWithFlags(&rt->side_join, cudaEventDisableTiming));
            }
            ULLIS_CUDA_CHECK(cudaEventRecord(rt->side_fork, rt->stream));
            ULLIS_CUDA_CHECK(cudaStreamWaitEvent(rt->side_stream, rt->side_fork, 0));
            // side_join must be recorded behind whatever reached the side stream, also when a step below throws
            struct Recorder {
                ullis_cuda_runtime* rt;
                SideJoin* side;
                ~Recorder() {
                    if (cudaEventRecord(rt->side_join, rt->side_stream) == cudaSuccess) side->forked = true;
                }
            };
            Recorder recorder{rt, &side};
            if (rt->kernel_timing) rt->side_begin();
            rosa_constq_kernel<<<cgrid, 128, 0, rt->side_stream>>>(q_sw, k_sw, v_sw, idx_sw, (uint32_t)time, wps, cq_list,
                                                                   cq_count);
            const cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) fail(ULLIS_CUDA_ERR_CUDA, std::string("launch of rosa_constq: ") + cudaGetErrorString(e));
            ++rt->launches;
            if (rt->kernel_timing) rt->side_end("rosa_constq");
        } else {
            rosa_constq_kernel<<<cgrid, 128, 0, rt->stream>>>(q_sw, k_sw, v_sw, idx_sw, (uint32_t)time, wps, cq_list, cq_count);
            rt->launched("rosa_constq");
        }
    }
    if (use_coop && !rt->sam_coop_ready) {
#define ULLIS_COOP_SMEM(NT, MODE) \
    ULLIS_CUDA_CHECK(cudaFuncSetAttribute(rosa_coop_kernel<NT, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024))
        ULLIS_COOP_SMEM(256, 0); ULLIS_COOP_SMEM(512, 0); ULLIS_COOP_SMEM(1024, 0);
        ULLIS_COOP_SMEM(256, 1); ULLIS_COOP_SMEM(512, 1); ULLIS_COOP_SMEM(1024, 1);
        ULLIS_COOP_SMEM(256, 2); ULLIS_COOP_SMEM(512, 2); ULLIS_COOP_SMEM(1024, 2);
#undef ULLIS_COOP_SMEM
        rt->sam_coop_ready = true;
    }
    for (size_t s0 = 0; s0 < streams; s0 += wave) {
        const size_t n = streams - s0 < wave ? streams - s0 : wave;
        const int lanes = rt->sam_lanes;
        const size_t warps = (n + lanes - 1) / lanes;
        const unsigned grid = (unsigned)((warps * 32 + 127) / 128);
        if (use_coop) {
            // sam_lanes_fixed: the caller pinned the streams per warp; otherwise the kernel picks 2 or 4
            const int pass1_lanes = rt->sam_lanes_fixed ? lanes : 0;
            const size_t pass1_warps = rt->sam_lanes_fixed ? warps : n;
            const unsigned p1_grid = (unsigned)((pass1_warps * 32 + 127) / 128);
            const uint32_t dense = 96u * (uint32_t)rt->sm_count, sparse = rt->sam_sparse_per_sm * (uint32_t)rt->sm_count;
            const bool split = rt->sam_split && rt->sam_words;
            const bool defer = !split && rt->sam_words && rt->sam_defer_climb;
            const int coop_mode = split ? 1 : defer ? 2 : 0;
            if (split) {
                rosa_extend_kernel<<<p1_grid, 128, 0, rt->stream>>>(scratch, stride, k_sw, list, count, s0, n,
                                                                   (uint32_t)time, wps, pass1_lanes, dense, sparse);
                rt->launched("rosa_extend");
                if (rt->sam_walk_chunked) {
                    rosa_walk_chunked_kernel<<<(unsigned)(((n + 3) / 4 * 32 + 127) / 128), 128, 0, rt->stream>>>(
                        scratch, stride, q_sw, list, count, s0, n, (uint32_t)time, wps);
                } else {
                    rosa_walk_kernel<<<p1_grid, 128, 0, rt->stream>>>(scratch, stride, q_sw, list, count, s0, n,
                                                                     (uint32_t)time, wps, pass1_lanes, dense, sparse);
                }
                rt->launched("rosa_walk");
            } else {
                // Few streams: the state arrays in shared memory, one one-warp CTA per stream, all resident at once.
                // How many streams reach the automaton is known on the device only, so the choice goes by what the
                // same call site (`site`: the model's layer) saw the last time its kernel ran - the kernels leave
                // that number in pinned host memory - and only when it was well inside one round of resident CTAs.
                // Either kernel is correct for any number of streams; a wrong guess costs time, not results.
                const size_t state_bytes = (size_t)sam::node_capacity((uint32_t)time) * sizeof(sam::Node<uint16_t>);
                uint32_t* hint = rt->sam_hint_slot(site);
                bool in_smem = false;
                if (defer && rt->sam_reload_w && rt->sam_smem_waves > 0 && hint && wave == streams &&
                    state_bytes <= 226 * 1024) {
                    const size_t per_sm = std::min<size_t>(32, (227 * 1024) / (state_bytes + 1024));
                    const size_t resident = per_sm * (size_t)rt->sm_count * (size_t)rt->sam_smem_waves;
                    const uint32_t expected = *static_cast<volatile uint32_t*>(hint);
                    in_smem = rt->sam_smem_waves >= 1000 || (expected != 0xFFFFFFFFu && (size_t)expected + expected / 8 <= resident);
                }
                if (in_smem) {
                    if (!rt->sam_smem_ready) {   // the attribute belongs to the function, not to this runtime: always the same value
                        ULLIS_CUDA_CHECK(cudaFuncSetAttribute(rosa_pass1_smem_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                              226 * 1024));
                        rt->sam_smem_ready = true;
                    }
                    rosa_pass1_smem_kernel<<<(unsigned)n, 32, state_bytes, rt->stream>>>(scratch, stride, q_sw, k_sw, list, count,
                                                                                        s0, n, (uint32_t)time, wps, hint);
                    rt->launched("rosa_pass1_smem");
                } else {
#define ULLIS_PASS1(W) \
    rosa_pass1_kernel<W><<<p1_grid, 128, 0, rt->stream>>>(scratch, stride, q_sw, k_sw, list, count, s0, n, (uint32_t)time, \
                                                          wps, pass1_lanes, dense, sparse, hint)
                if (!rt->sam_words) ULLIS_PASS1(0);
                else if (defer && rt->sam_reload_w) ULLIS_PASS1(3);
                else if (defer) ULLIS_PASS1(2);
                else ULLIS_PASS1(1);
#undef ULLIS_PASS1
                rt->launched("rosa_pass1");
                }
            }
            // threads per stream: the fewer CTAs shared memory lets an SM hold, the more threads each one gets
            const unsigned coop_per_sm = (unsigned)((227u * 1024u) / (coop.total + 1024u));
            const int coop_threads = rt->sam_coop_threads ? rt->sam_coop_threads : coop_per_sm >= 3 ? 256 : coop_per_sm == 2 ? 512 : 1024;
#define ULLIS_COOP_LAUNCH_MODE(NT, MODE)                                                                                 \
    rosa_coop_kernel<NT, MODE><<<(unsigned)n, NT, coop.total, rt->stream>>>(scratch, stride, v_sw, idx_sw, list, count, s0, \
                                                                            (uint32_t)time, wps, rt->dev_status)
#define ULLIS_COOP_LAUNCH(NT)                                 \
    do {                                                      \
        if (coop_mode == 1) ULLIS_COOP_LAUNCH_MODE(NT, 1);    \
        else if (coop_mode == 2) ULLIS_COOP_LAUNCH_MODE(NT, 2); \
        else ULLIS_COOP_LAUNCH_MODE(NT, 0);                   \
    } while (0)
            if (coop_threads == 256) ULLIS_COOP_LAUNCH(256);
            else if (coop_threads == 512) ULLIS_COOP_LAUNCH(512);
            else ULLIS_COOP_LAUNCH(1024);
#undef ULLIS_COOP_LAUNCH_MODE
#undef ULLIS_COOP_LAUNCH
            rt->launched("rosa_coop");
            continue;
        }
#define ULLIS_SAM_LAUNCH(IX, ALGO)                                                                              \
    rosa_sam_kernel<IX, ALGO><<<grid, 128, 0, rt->stream>>>(scratch, stride, q_sw, k_sw, v_sw, idx_sw, list, count, s0, \
                                                           n, (uint32_t)time, wps, lanes, rt->dev_status)
        if (narrow) {
            if (algo == ULLIS_CUDA_SAM_EAGER) ULLIS_SAM_LAUNCH(uint16_t, ULLIS_CUDA_SAM_EAGER);
            else ULLIS_SAM_LAUNCH(uint16_t, ULLIS_CUDA_SAM_EULER);
        } else {
            if (algo == ULLIS_CUDA_SAM_EAGER) ULLIS_SAM_LAUNCH(uint32_t, ULLIS_CUDA_SAM_EAGER);
            else ULLIS_SAM_LAUNCH(uint32_t, ULLIS_CUDA_SAM_EULER);
        }
#undef ULLIS_SAM_LAUNCH
        rt->launched("rosa_sam");
    }
    // `side` goes out of scope here: `stream` waits for the side kernel, idx is complete on `stream` from then on
}

}  // namespace k
}  // namespace ullis
