// Host side of the tensor-core stages: TMA descriptors, the small kernels that
// prepare 16-bit operands (time-shift mixes with a hi+lo FP16 split, +/-e
// emit, f32 -> 16-bit casts), the exact fix-up of sign bits that fall inside
// the tensor-core error band, the CE finishing reduction, and the launch of
// the tcgen05 GEMM (tc_gemm.cuh) with the epilogue each stage needs.
#include "linear_tc.hpp"

#include <cudaTypedefs.h>

#include <algorithm>
#include <cstring>

#include "kernels.hpp"
#include "tc_gemm.cuh"
#include "tc_gemm_ws.cuh"
#include "tc_gemm_ws2.cuh"

namespace ullis {
namespace tc {

namespace {

// ------------------------------------------------------------ TMA descriptors
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        ULLIS_CUDA_CHECK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
        if (!p || q != cudaDriverEntryPointSuccess) fail(ULLIS_CUDA_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable");
        fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

// [rows, K] 16-bit row-major matrix, boxes of 64 columns x 128 rows (or fewer), 128-byte swizzle, zero fill
CUtensorMap make_map(const void* ptr, size_t rows, size_t K, bool bf16, uint32_t box_rows = BM) {
    CUtensorMap m;
    cuuint64_t dims[2] = {K, rows};
    cuuint64_t strides[1] = {K * 2};
    cuuint32_t box[2] = {BK, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = encode_fn()(&m, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                             const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) fail(ULLIS_CUDA_ERR_CUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
    return m;
}

__device__ __forceinline__ float h2f(uint16_t b) { return __half2float(__ushort_as_half(b)); }

// ------------------------------------------------------------ operand kernels
// f32 -> f16 / bf16
// (FP16 ends at 65504: a larger finite input is reported through the status word, not turned into inf)
__global__ void cast16_kernel(const float* __restrict__ x, uint16_t* __restrict__ y, size_t n, int bf16, size_t K,
                              uint32_t* __restrict__ status) {
    chain_entry();
    size_t e = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (e >= n) return;
    float v[4];
    for (int k = 0; k < 4; ++k) v[k] = e + k < n ? x[e + k] : 0.0f;
    for (int k = 0; k < 4; ++k) {
        if (e + k >= n) break;
        if (!bf16 && fabsf(v[k]) > 65504.0f && fabsf(v[k]) <= 3.4028234e38f &&
            atomicCAS(status, ULLIS_DEV_OK, ULLIS_DEV_FP16_RANGE) == ULLIS_DEV_OK)
            status[1] = (uint32_t)((e + k) / K);
        y[e + k] = bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v[k])) : __half_as_ushort(__float2half_rn(v[k]));
    }
}

// Time-shift mixes of one LayerNorm output (reference src/model.rs:1291-1298:
// in = x + (x[t-1]-x[t])*mix, unfused) written as FP16 hi and lo = FP16(in - hi)
// for up to three mixes, plus the row's sum |in| that scales the sign-bit error
// band. One warp per row.  A sequence of `time` rows takes `pitch` rows of the operands (and of s1): the sign-bit
// GEMM wants the steps of a sequence in whole words; what is in the rows between is never looked at.
__global__ void __launch_bounds__(256)
mix_split_kernel(const float* __restrict__ x, const uint16_t* __restrict__ m0, const uint16_t* __restrict__ m1,
                 const uint16_t* __restrict__ m2, uint16_t* __restrict__ hi0, uint16_t* __restrict__ lo0,
                 uint16_t* __restrict__ hi1, uint16_t* __restrict__ lo1, uint16_t* __restrict__ hi2,
                 uint16_t* __restrict__ lo2, float* __restrict__ s1, size_t rows, size_t time, size_t pitch, size_t C) {
    chain_entry();
    const int lane = threadIdx.x & 31;
    const size_t row = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const bool first = row % time == 0;
    const size_t orow = row + row / time * (pitch - time), orows = rows / time * pitch;
    const uint16_t* mix[3] = {m0, m1, m2};
    uint16_t* hi[3] = {hi0, hi1, hi2};
    uint16_t* lo[3] = {lo0, lo1, lo2};
    float sum[3] = {0.0f, 0.0f, 0.0f};
    // four channels per lane and step (C % 4 == 0 on this path): 16-byte loads, 8-byte stores
    for (size_t c = (size_t)lane * 4; c < C; c += 128) {
        const float4 cur = *reinterpret_cast<const float4*>(x + row * C + c);
        float4 prev = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!first) prev = *reinterpret_cast<const float4*>(x + (row - 1) * C + c);
        const float xt[4] = {cur.x, cur.y, cur.z, cur.w}, pt[4] = {prev.x, prev.y, prev.z, prev.w};
        float xx[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) xx[e] = first ? -xt[e] : __fsub_rn(pt[e], xt[e]);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (!mix[k]) continue;
            const uint2 mw = *reinterpret_cast<const uint2*>(mix[k] + c);
            const uint16_t mb[4] = {(uint16_t)(mw.x & 0xFFFFu), (uint16_t)(mw.x >> 16), (uint16_t)(mw.y & 0xFFFFu),
                                    (uint16_t)(mw.y >> 16)};
            uint16_t hb[4], lb[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float v = __fadd_rn(xt[e], __fmul_rn(xx[e], h2f(mb[e])));
                const __half h = __float2half_rn(v);
                hb[e] = __half_as_ushort(h);
                lb[e] = __half_as_ushort(__float2half_rn(v - __half2float(h)));
                sum[k] += fabsf(v);
            }
            *reinterpret_cast<uint2*>(hi[k] + orow * C + c) =
                make_uint2(hb[0] | ((uint32_t)hb[1] << 16), hb[2] | ((uint32_t)hb[3] << 16));
            if (lo[k])
                *reinterpret_cast<uint2*>(lo[k] + orow * C + c) =
                    make_uint2(lb[0] | ((uint32_t)lb[1] << 16), lb[2] | ((uint32_t)lb[3] << 16));
        }
    }
    if (s1) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            float s = sum[k];
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0 && mix[k]) s1[k * orows + orow] = s;
        }
    }
}

// LayerNorm and mix_split_kernel in one pass over the residual stream: a warp normalises its row and the row
// before it (the same arithmetic as the stand-alone warp LayerNorm, so both warps that need a row get the same
// values), forms the mixes and writes the 16-bit operands; the LayerNorm output itself is only written when
// something downstream reads it as f32 (`ln_out`: the exact sign fix-up).  Saves the round trip of the
// LayerNorm output through HBM.  C = 128 * VEC channels, VEC <= 8.
// A warp takes one row, or (SEVERAL) `per_warp` consecutive ones: the LayerNorm of a row is then computed once and handed
// on as the next row's "row before" (with one every row is normalised twice, by its own warp and by its successor's).
// MIXES = 1: one operand in 16 bits alone (m0 -> hi0; no lo, s1, ln_out).
// Bound by memory for many rows and by a warp's chain of load, two reductions and store for few: everything the rows
// share is loaded with the first row, and a row's loads go out before the row before it is worked on.
template <int VEC, bool SEVERAL, int MIXES>
__global__ void __launch_bounds__(256, VEC <= 4 ? 2 : 1)
ln_mix_split_kernel(const float* __restrict__ x, const uint16_t* __restrict__ lw, const uint16_t* __restrict__ lb,
                    float* __restrict__ ln_out, const uint16_t* __restrict__ m0, const uint16_t* __restrict__ m1,
                    const uint16_t* __restrict__ m2, uint16_t* __restrict__ hi0, uint16_t* __restrict__ lo0,
                    uint16_t* __restrict__ hi1, uint16_t* __restrict__ lo1, uint16_t* __restrict__ hi2,
                    uint16_t* __restrict__ lo2, float* __restrict__ s1, uint32_t rows, uint32_t time, uint32_t pitch,
                    uint32_t per_warp) {
    chain_entry();
    constexpr int C = 128 * VEC;
    // as far as the registers go
    constexpr bool AHEAD = SEVERAL && VEC <= 4, MIX_FIRST = VEC <= 4 && (MIXES == 1 || !SEVERAL);
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t row0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (SEVERAL ? per_warp : 1u);
    if (row0 >= rows) return;
    const uint32_t last = SEVERAL ? min(row0 + per_warp, rows) : row0 + 1;
    const uint16_t* mix[3] = {m0, m1, m2};
    uint16_t* hi[3] = {hi0, hi1, hi2};
    uint16_t* lo[3] = {lo0, lo1, lo2};
    uint32_t seq = row0 / time, step = row0 - seq * time;
    float4 cur[VEC], prev[VEC], next[VEC];
    uint2 w[VEC], b[VEC], m[MIXES][VEC];
    const auto load_row = [&](float4 (&v)[VEC], uint32_t row) {
        const float4* src = reinterpret_cast<const float4*>(x + (size_t)row * C) + lane;
#pragma unroll
        for (int i = 0; i < VEC; ++i) v[i] = src[32 * i];
    };
    load_row(cur, row0);
#pragma unroll
    for (int i = 0; i < VEC; ++i) prev[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (step) load_row(prev, row0 - 1);
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
        w[i] = reinterpret_cast<const uint2*>(lw)[lane + 32 * i];
        b[i] = reinterpret_cast<const uint2*>(lb)[lane + 32 * i];
#pragma unroll
        for (int k = 0; k < MIXES; ++k)
            if (MIX_FIRST) m[k][i] = reinterpret_cast<const uint2*>(mix[k])[lane + 32 * i];
    }
    // normalised values of one row, in place
    const auto layer_norm_row = [&](float4 (&v)[VEC]) {
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < VEC; ++i) sum += (v[i].x + v[i].y) + (v[i].z + v[i].w);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        const float mean = sum / (float)C;
        float sq = 0.0f;
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
            float a = v[i].x - mean, bb = v[i].y - mean, c = v[i].z - mean, d = v[i].w - mean;
            sq += (a * a + bb * bb) + (c * c + d * d);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        const float inv = 1.0f / sqrtf(sq / (float)C + 1e-5f);
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
            v[i].x = (v[i].x - mean) * inv * h2f((uint16_t)(w[i].x & 0xffff)) + h2f((uint16_t)(b[i].x & 0xffff));
            v[i].y = (v[i].y - mean) * inv * h2f((uint16_t)(w[i].x >> 16)) + h2f((uint16_t)(b[i].x >> 16));
            v[i].z = (v[i].z - mean) * inv * h2f((uint16_t)(w[i].y & 0xffff)) + h2f((uint16_t)(b[i].y & 0xffff));
            v[i].w = (v[i].w - mean) * inv * h2f((uint16_t)(w[i].y >> 16)) + h2f((uint16_t)(b[i].y >> 16));
        }
    };
    layer_norm_row(prev);   // of a sequence's first step: not used
#pragma unroll 1
    for (uint32_t row = row0; row < last; ++row) {
        if (AHEAD && row + 1 < last) load_row(next, row + 1);
        const bool first = step == 0;   // the same for the whole warp
        const size_t orow = (size_t)seq * pitch + step;
        layer_norm_row(cur);
        if (MIXES > 1 && ln_out) {
            float4* dst = reinterpret_cast<float4*>(ln_out + (size_t)row * C) + lane;
#pragma unroll
            for (int i = 0; i < VEC; ++i) dst[32 * i] = cur[i];
        }
        float sum[MIXES] = {};
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
            const float xt[4] = {cur[i].x, cur[i].y, cur[i].z, cur[i].w};
            const float pt[4] = {prev[i].x, prev[i].y, prev[i].z, prev[i].w};
            float xx[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) xx[e] = first ? -xt[e] : __fsub_rn(pt[e], xt[e]);
#pragma unroll
            for (int k = 0; k < MIXES; ++k) {
                if (!MIX_FIRST) m[k][i] = reinterpret_cast<const uint2*>(mix[k])[lane + 32 * i];
                const uint32_t mb[4] = {m[k][i].x & 0xFFFFu, m[k][i].x >> 16, m[k][i].y & 0xFFFFu, m[k][i].y >> 16};
                float v[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    v[e] = __fadd_rn(xt[e], __fmul_rn(xx[e], h2f((uint16_t)mb[e])));
                    if (MIXES > 1) sum[k] += fabsf(v[e]);
                }
                const size_t at = orow * C + (lane + 32 * i) * 4;
                const __half2 h01 = __floats2half2_rn(v[0], v[1]), h23 = __floats2half2_rn(v[2], v[3]);
                *reinterpret_cast<uint2*>(hi[k] + at) =
                    make_uint2(*reinterpret_cast<const uint32_t*>(&h01), *reinterpret_cast<const uint32_t*>(&h23));
                if (MIXES > 1) {
                    const float2 f01 = __half22float2(h01), f23 = __half22float2(h23);
                    const __half2 l01 = __floats2half2_rn(v[0] - f01.x, v[1] - f01.y);
                    const __half2 l23 = __floats2half2_rn(v[2] - f23.x, v[3] - f23.y);
                    *reinterpret_cast<uint2*>(lo[k] + at) =
                        make_uint2(*reinterpret_cast<const uint32_t*>(&l01), *reinterpret_cast<const uint32_t*>(&l23));
                }
            }
        }
        if (MIXES > 1) {
#pragma unroll
            for (int k = 0; k < MIXES; ++k) {
                float s = sum[k];
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (lane == 0) s1[(size_t)k * (rows / time * pitch) + orow] = s;
            }
        }
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
            prev[i] = cur[i];
            if (AHEAD) cur[i] = next[i];
        }
        if (SEVERAL && !AHEAD && row + 1 < last) load_row(cur, row + 1);
        if (++step == time) {
            step = 0;
            ++seq;
        }
    }
}

// idx bits (stream-major) -> y = +/-e as FP16 [B*T, C] (reference src/model.rs:1313)
// One CTA: 32 steps x 256 channels; a thread writes eight channels (16 bytes) of four steps.
__global__ void __launch_bounds__(256)
emit_f16_kernel(const uint32_t* __restrict__ idx_sw, const uint16_t* __restrict__ e, uint16_t* __restrict__ y,
                size_t T, size_t C, size_t wps) {
    chain_entry();
    __shared__ __align__(16) uint32_t wsm[256];
    const size_t b = blockIdx.z, t0 = (size_t)blockIdx.x * 32, c0 = (size_t)blockIdx.y * 256;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    wsm[threadIdx.x] = (c0 + threadIdx.x < C) ? idx_sw[(b * C + c0 + threadIdx.x) * wps + blockIdx.x] : 0u;
    __syncthreads();
    const size_t c = c0 + (size_t)tx * 8;
    if (c >= C) return;   // C % 8 == 0 on this path
    const uint4 ev = *reinterpret_cast<const uint4*>(e + c);
    const uint32_t eb[8] = {ev.x & 0xFFFFu, ev.x >> 16, ev.y & 0xFFFFu, ev.y >> 16,
                            ev.z & 0xFFFFu, ev.z >> 16, ev.w & 0xFFFFu, ev.w >> 16};
    const uint4 wa = reinterpret_cast<const uint4*>(wsm)[tx * 2], wb = reinterpret_cast<const uint4*>(wsm)[tx * 2 + 1];
    const uint32_t words[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t tt = ty * 4 + k;
        if (t0 + tt >= T) break;
        uint32_t h[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) h[j] = eb[j] ^ (((words[j] >> tt) & 1u) ? 0u : 0x8000u);  // flip the FP16 sign for idx 0
        *reinterpret_cast<uint4*>(y + (b * T + t0 + tt) * C + c) =
            make_uint4(h[0] | (h[1] << 16), h[2] | (h[3] << 16), h[4] | (h[5] << 16), h[6] | (h[7] << 16));
    }
}

// Exact pre-activation sign of one output of a packed linear over the time-shift mix of x, as the reference
// computes it (src/model.rs:1291-1298 then 724-742): in_i = x_i + (x[t-1]_i - x_i) * mix_i (unfused), the sum of
// +/- in_i for i ascending in f32, then bias + scale * sum.  R inputs per round: the 2R/4 row loads of a round go
// out together, then the sum is taken in order.
template <int R>
__device__ __forceinline__ bool exact_mixed_sign(const float* __restrict__ xr, bool first_step,
                                                 const uint16_t* __restrict__ mix, const uint32_t* __restrict__ wbits,
                                                 float scale, float bias, size_t C) {
    float sum = 0.0f;
    for (size_t i0 = 0; i0 < C; i0 += R) {
        float4 cur[R / 4], prev[R / 4];
#pragma unroll
        for (int u = 0; u < R / 4; ++u) {
            cur[u] = *reinterpret_cast<const float4*>(xr + i0 + 4 * u);
            prev[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!first_step) prev[u] = *reinterpret_cast<const float4*>(xr - C + i0 + 4 * u);
        }
        const uint32_t wword = wbits[i0 >> 5] >> (i0 & 31);
#pragma unroll
        for (int u = 0; u < R / 4; ++u) {
            const float xs[4] = {cur[u].x, cur[u].y, cur[u].z, cur[u].w};
            const float ps[4] = {prev[u].x, prev[u].y, prev[u].z, prev[u].w};
            const uint2 mw = *reinterpret_cast<const uint2*>(mix + i0 + 4 * u);
            const uint16_t mb[4] = {(uint16_t)(mw.x & 0xFFFFu), (uint16_t)(mw.x >> 16), (uint16_t)(mw.y & 0xFFFFu),
                                    (uint16_t)(mw.y >> 16)};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float xt = xs[k];
                const float xx = first_step ? -xt : __fsub_rn(ps[k], xt);
                const float in = __fadd_rn(xt, __fmul_rn(xx, h2f(mb[k])));
                sum = __fmaf_rn((wword >> (4 * u + k)) & 1u ? 1.0f : -1.0f, in, sum);
            }
        }
    }
    return __fadd_rn(bias, __fmul_rn(scale, sum)) > 0.0f;
}

// The exact recomputation of the flagged outputs of a Q/K/V launch, a CTA per (sequence, block of 32 steps) or per `steps` of
// one (4, 8, 16): the sequential f32 sum of the reference (src/model.rs:724-742) is a chain that only one thread can run, and all
// entries of a block (about 50 with 512 channels) read the same 33 rows of x.  So the rows come to shared memory once, 64 columns
// at a time with the next 64 on their way, and a thread has an entry.  Entries are sorted by step, so that eight lanes side by side
// read few rows that follow on each other, and 16 bytes of each meet no bank conflict.  Where a sequence begins the row before is
// 0, since 0 - x is -x up to the sign of a zero, which the sum with x does away with.
// With few blocks bound by the chain, with many by the waits for rows and at the barriers: issue slots 39 % used at 16 sequences, 30 %
// of the warps there (a third buffer 110 -> 128 us, fewer blocks per SM; one barrier per 64 columns instead of two 110 -> 115).
// Unsorted, with 4-byte copies and reads, a warp issued three times as much.  64 sequences of the default model, us per layer: a kernel that
// listed the entries, one that read both rows of each anew for its warp, 4 KB per entry through L2, and one that left at once 179,
// so 110.  The whole call: 64 sequences 26 860 -> 26 080, 16 in training 11 540 -> 11 370, 5 x 1531 3 697 -> 3 607, one
// 2 215 -> 2 183.
// Whole rows at once where a CTA has few steps, without the waits in between, took the kernel from 12.7 to 11.4 us a layer by itself and one
// sequence from 1 817 to 1 844 us.
// Any number of flags: what the queue does not hold waits in its finder's registers.
constexpr uint32_t FIXB_COLS = 64, FIXB_PITCH = FIXB_COLS + 4, FIXB_ROWS = 33, FIXB_QUEUE = 512, FIXB_WORDS = 8, FIXB_MAX_THREADS = 160;
// Threads per CTA: a third more than there are entries on average, so that hardly a block needs a second round; at most
// FIXB_WORDS flag words of a matrix for each.
inline unsigned fix_block_threads(size_t C) { return 32u * (unsigned)((C + 32 * FIXB_WORDS - 1) / (32 * FIXB_WORDS) + 1); }
inline size_t fix_block_smem(size_t C) { return 4 * (3 * (C + 4) + 2 * FIXB_ROWS * FIXB_PITCH + FIXB_QUEUE); }

__global__ void __launch_bounds__(FIXB_MAX_THREADS)
fix_block_kernel(const float* __restrict__ x, const uint16_t* __restrict__ mq, const uint16_t* __restrict__ mk,
                 const uint16_t* __restrict__ mv, PackedWeights wq, PackedWeights wk, PackedWeights wv,
                 uint32_t* __restrict__ bq, uint32_t* __restrict__ bk, uint32_t* __restrict__ bv,
                 const uint32_t* __restrict__ flags, size_t sw, uint32_t T, uint32_t C, uint32_t wps, uint32_t steps) {
    extern __shared__ __align__(16) float fix_mem[];
    float* mixes = fix_mem;                                     // [3][C + 4]
    float* rows = mixes + 3 * (C + 4);                          // [2][FIXB_ROWS][FIXB_PITCH]
    uint32_t* queue = reinterpret_cast<uint32_t*>(rows + 2 * FIXB_ROWS * FIXB_PITCH);
    __shared__ uint32_t places[32], found;   // per step: entries, then where the next one goes
    const uint32_t tid = threadIdx.x, nt = blockDim.x;
    for (uint32_t c = tid; c < C; c += nt) {
        mixes[c] = h2f(mq[c]);
        mixes[C + 4 + c] = h2f(mk[c]);
        mixes[2 * (C + 4) + c] = h2f(mv[c]);
    }
    if (tid < 32) places[tid] = 0;
    chain_entry();   // the mixes are weights, which the kernel directly before never writes
    const uint32_t of = blockIdx.x * steps / 32u, b = of / wps, word = of - b * wps, s0 = blockIdx.x * steps % 32u, t0 = word * 32u + s0;
    const uint32_t have = t0 < T ? min(steps, T - t0) : 0u, mask = (~0u >> (32u - steps)) << s0;   // no flags past T
    const float* block = x + ((size_t)b * T + t0) * C;
    const uint32_t* of_block = flags + (size_t)of * C;   // channels side by side, a matrix every sw words
    uint32_t f[3][FIXB_WORDS];
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (uint32_t u = 0; u < FIXB_WORDS; ++u) f[m][u] = u * nt + tid < C ? of_block[m * sw + u * nt + tid] & mask : 0u;
    const auto fetch = [&](uint32_t chunk) {
        float* to = rows + (chunk & 1u) * (FIXB_ROWS * FIXB_PITCH);
        const float* from = block + chunk * FIXB_COLS;
        for (uint32_t i = tid; i < (steps + 1u) * (FIXB_COLS / 4); i += nt) {
            const uint32_t r = i / (FIXB_COLS / 4), c = i % (FIXB_COLS / 4) * 4;   // row r is step t0 + r - 1
            float* slot = to + r * FIXB_PITCH + c;
            if (r ? r <= have : t0 != 0u)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(slot)),
                             "l"(from + (ptrdiff_t)r * C - C + c) : "memory");
            else
                *reinterpret_cast<float4*>(slot) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const uint32_t chunks = C / FIXB_COLS;
    const auto drain = [&](uint32_t count) {
        for (uint32_t e0 = 0; e0 < count; e0 += nt) {
            const bool live = e0 + tid < count;
            const uint32_t entry = live ? queue[e0 + tid] : s0, tt = entry & 31u, ch = (entry >> 5) & 0x7FFFFFu, m = entry >> 28;
            const uint32_t* w = (m == 0u ? wq.bits : m == 1u ? wk.bits : wv.bits) + ((size_t)ch * C >> 5);   // C % 64 == 0
            uint32_t signs[2] = {w[0], w[1]};
            const float* mix = mixes + m * (C + 4);
            float sum = 0.0f;
            fetch(0);
#pragma unroll 1
            for (uint32_t k = 0; k < chunks; ++k) {
                uint32_t ahead[2] = {0u, 0u};
                if (k + 1 < chunks) {
                    fetch(k + 1);
                    ahead[0] = w[2 * k + 2];
                    ahead[1] = w[2 * k + 3];
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                } else {
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                }
                __syncthreads();
                const float* prev = rows + (k & 1u) * (FIXB_ROWS * FIXB_PITCH) + (tt - s0) * FIXB_PITCH;
                if (live) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
#pragma unroll
                        for (int j = 0; j < 32; j += 4) {   // i ascending
                            const float4 mw = *reinterpret_cast<const float4*>(mix + k * FIXB_COLS + 32 * h + j);
                            const float4 before = *reinterpret_cast<const float4*>(prev + 32 * h + j);
                            const float4 at = *reinterpret_cast<const float4*>(prev + FIXB_PITCH + 32 * h + j);
                            const float mv4[4] = {mw.x, mw.y, mw.z, mw.w}, ps[4] = {before.x, before.y, before.z, before.w};
                            const float xs[4] = {at.x, at.y, at.z, at.w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const float in = __fadd_rn(xs[e], __fmul_rn(__fsub_rn(ps[e], xs[e]), mv4[e]));
                                const uint32_t flip = (~signs[h] << (31 - j - e)) & 0x80000000u;   // bit set: +
                                sum = __fadd_rn(sum, __uint_as_float(__float_as_uint(in) ^ flip));
                            }
                        }
                    }
                }
                signs[0] = ahead[0];
                signs[1] = ahead[1];
                __syncthreads();   // this half of `rows` is filled anew two chunks on
            }
            if (live) {
                const uint16_t* scale = m == 0u ? wq.scale : m == 1u ? wk.scale : wv.scale;
                const uint16_t* bias = m == 0u ? wq.bias : m == 1u ? wk.bias : wv.bias;
                const float y = __fadd_rn(bias ? h2f(bias[ch]) : 0.0f, __fmul_rn(h2f(scale[ch]), sum));
                uint32_t* at = (m == 0u ? bq : m == 1u ? bk : bv) + ((size_t)b * C + ch) * wps + word;
                if (y > 0.0f) atomicOr(at, 1u << tt); else atomicAnd(at, ~(1u << tt));
            }
        }
    };
    __syncthreads();   // `places` are 0
    for (;;) {
#pragma unroll
        for (int m = 0; m < 3; ++m)
#pragma unroll
            for (uint32_t u = 0; u < FIXB_WORDS; ++u)
                for (uint32_t g = f[m][u]; g; g &= g - 1u) atomicAdd(&places[__ffs(g) - 1], 1u);
        __syncthreads();
        if (tid < 32) {
            const uint32_t n = places[tid];
            uint32_t up_to = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t other = __shfl_up_sync(0xFFFFFFFFu, up_to, o);
                if (tid >= (uint32_t)o) up_to += other;
            }
            places[tid] = up_to - n;
            if (tid == 31) found = up_to;
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < 3; ++m)
#pragma unroll
            for (uint32_t u = 0; u < FIXB_WORDS; ++u)
                for (uint32_t g = f[m][u]; g; g &= g - 1u) {
                    const uint32_t step = __ffs(g) - 1, at = atomicAdd(&places[step], 1u);
                    if (at >= FIXB_QUEUE) continue;
                    queue[at] = (uint32_t)m << 28 | (u * nt + tid) << 5 | step;
                    f[m][u] &= ~(1u << step);
                }
        const uint32_t n = found;
        __syncthreads();
        drain(min(n, FIXB_QUEUE));
        if (n <= FIXB_QUEUE) return;
        __syncthreads();
        if (tid < 32) places[tid] = 0;
        __syncthreads();
    }
}

// Sign bits whose tensor-core pre-activation fell inside the error band are
// recomputed exactly as the reference does (src/model.rs:724-742 on the
// time-shift mix of x): sequential f32 sum over i, then bias + scale*sum.
// Flags are sparse (a few per thousand).  A CTA owns a window of 64 steps of
// one sequence for ALL channels of Q, K and V, so the 65 rows of x its exact
// dot products read stay in L1 / L2 and every row is fetched from HBM about
// once per launch; it gathers the flagged (matrix, channel, step) triples into
// a shared queue and spreads them over its threads, one dot product each.
constexpr int FIX_THREADS = 256, FIX_WIN = 2 /* flag words (of 32 steps) per window */, FIX_QUEUE = 12288, FIX_BATCH = 8;
static_assert(FIX_QUEUE >= FIX_THREADS * 32, "the flag bits of one word per thread must fit the queue");

__global__ void __launch_bounds__(FIX_THREADS)
sign_fixup_kernel(const float* __restrict__ x, const uint16_t* __restrict__ mq, const uint16_t* __restrict__ mk,
                  const uint16_t* __restrict__ mv, PackedWeights wq, PackedWeights wk, PackedWeights wv,
                  uint32_t* __restrict__ bq, uint32_t* __restrict__ bk, uint32_t* __restrict__ bv,
                  const uint32_t* __restrict__ fq, const uint32_t* __restrict__ fk, const uint32_t* __restrict__ fv,
                  size_t batch, size_t T, size_t C, size_t wps) {
    chain_entry();
    extern __shared__ uint32_t fix_queue[];  // entries: matrix << 28 | channel << 8 | word in window << 5 | bit
    __shared__ uint32_t q_count, announced;   // entries queued; flag bits announced so far (never reset)
    const size_t windows = (wps + FIX_WIN - 1) / FIX_WIN;
    const size_t b = blockIdx.x / windows, w0 = (blockIdx.x % windows) * FIX_WIN;
    const uint32_t per_matrix = (uint32_t)C * FIX_WIN, items = 3u * per_matrix;
    if (threadIdx.x == 0) { q_count = 0; announced = 0; }
    __syncthreads();

    // one exact dot product per queued entry, spread over the CTA's threads; empties the queue
    auto drain = [&]() {
        __syncthreads();
        const uint32_t count = q_count;
        for (uint32_t i = threadIdx.x; i < count; i += FIX_THREADS) {
            const uint32_t entry = fix_queue[i], tt = entry & 31u, m = entry >> 28;
            const size_t ch = (entry >> 8) & 0xFFFFFu, word = w0 + ((entry >> 5) & 7u);
            const size_t ew = (b * C + ch) * wps + word;
            const size_t t = word * 32 + tt, row = b * T + t;
            const float* xr = x + row * C;
            const uint16_t* mix = m == 0 ? mq : m == 1 ? mk : mv;
            const uint32_t* wb = m == 0 ? wq.bits : m == 1 ? wk.bits : wv.bits;
            const uint16_t* wscale = m == 0 ? wq.scale : m == 1 ? wk.scale : wv.scale;
            const uint16_t* wbias = m == 0 ? wq.bias : m == 1 ? wk.bias : wv.bias;
            uint32_t* bits = m == 0 ? bq : m == 1 ? bk : bv;
            const uint32_t* wbits = wb + (ch * C >> 5);  // C % 32 == 0 on this path
            const bool plus = exact_mixed_sign<32>(xr, t == 0, mix, wbits, h2f(wscale[ch]), wbias ? h2f(wbias[ch]) : 0.0f, C);
            if (plus) atomicOr(&bits[ew], 1u << tt); else atomicAnd(&bits[ew], ~(1u << tt));
        }
        __syncthreads();
        if (threadIdx.x == 0) q_count = 0;
        __syncthreads();
    };
    auto push = [&](uint32_t f, uint32_t it) {
        const uint32_t which = it / per_matrix, rem = it % per_matrix;
        const uint32_t at = atomicAdd(&q_count, (uint32_t)__popc(f));
        uint32_t k = 0;
        while (f) {
            const uint32_t tt = __ffs(f) - 1;
            f &= f - 1;
            fix_queue[at + k++] = which << 28 | (rem / FIX_WIN) << 8 | (rem % FIX_WIN) << 5 | tt;
        }
    };

    // Flag words are read FIX_BATCH per thread at a time, all loads in flight together; the CTA first
    // announces how many bits the batch holds so that every thread takes the same decision about the queue.
    uint32_t seen = 0;   // value of `announced` before this batch (the same in every thread)
    for (uint32_t base = 0; base < items; base += FIX_THREADS * FIX_BATCH) {
        uint32_t f[FIX_BATCH], mine = 0;
#pragma unroll
        for (int k = 0; k < FIX_BATCH; ++k) {
            const uint32_t it = base + k * FIX_THREADS + threadIdx.x;
            f[k] = 0;
            if (it < items) {
                const uint32_t which = it / per_matrix, rem = it % per_matrix;
                const uint32_t* flags = which == 0 ? fq : which == 1 ? fk : fv;
                const size_t word = w0 + rem % FIX_WIN;
                if (word < wps) f[k] = flags[(b * wps + word) * C + rem / FIX_WIN];
            }
        }
#pragma unroll
        for (int k = 0; k < FIX_BATCH; ++k) mine += (uint32_t)__popc(f[k]);
        if (mine) atomicAdd(&announced, mine);
        __syncthreads();
        const uint32_t batch_bits = announced - seen, queued = q_count;
        seen = announced;
        __syncthreads();   // everyone has read both counters before either moves again
        if (queued + batch_bits > FIX_QUEUE) drain();
        if (batch_bits <= FIX_QUEUE) {
#pragma unroll
            for (int k = 0; k < FIX_BATCH; ++k)
                if (f[k]) push(f[k], base + k * FIX_THREADS + threadIdx.x);
        } else {   // dense flags: one word per thread at a time (at most 32 * FIX_THREADS entries)
#pragma unroll
            for (int k = 0; k < FIX_BATCH; ++k) {
                if (f[k]) push(f[k], base + k * FIX_THREADS + threadIdx.x);
                drain();
            }
        }
    }
    drain();
}

// Merge the per-tile (max, sum exp) partials of a row and subtract the target
// logit (reference src/model.rs:3219-3227; valid-row rule 27-39).  A warp per row: bound by the latency of one trip to the
// partials, which a thread per row made 128 times one after the other, in as few blocks as 256 rows fill
// (with the launch: 512 rows of 128 partials 41 -> 6 us, 32 768 rows 41 -> 14).
__global__ void __launch_bounds__(256)
ce_finish_kernel(const float2* __restrict__ part, const float* __restrict__ target_logit,
                                 const uint32_t* __restrict__ labels, uint32_t ignore_id, size_t rows, size_t time,
                                 size_t vocab, uint32_t n_tiles, float* __restrict__ row_loss, uint32_t* status) {
    chain_entry();
    const uint32_t lane = threadIdx.x & 31u;
    const size_t m = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (m >= rows) return;
    const bool valid = time != 0 && (m % time) + 1 < time && m + 1 < rows && labels[m + 1] != ignore_id;
    if (!valid) {
        if (lane == 0) row_loss[m] = 0.0f;
        return;
    }
    if (labels[m + 1] >= vocab) {
        if (lane == 0) {
            if (atomicCAS(status, ULLIS_DEV_OK, ULLIS_DEV_BAD_TOKEN) == ULLIS_DEV_OK) status[1] = (uint32_t)m;
            row_loss[m] = 0.0f;
        }
        return;
    }
    const float2* of = part + m * n_tiles;
    float gmax = -INFINITY;
    for (uint32_t i = lane; i < n_tiles; i += 32u) gmax = fmaxf(gmax, of[i].x);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) gmax = fmaxf(gmax, __shfl_xor_sync(0xFFFFFFFFu, gmax, o));
    float sum = 0.0f;
    for (uint32_t i = lane; i < n_tiles; i += 32u) {
        const float2 pr = of[i];
        sum += pr.y * expf(pr.x - gmax);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    if (lane == 0) row_loss[m] = gmax + logf(sum) - target_logit[m];
}

inline unsigned blocks_for(size_t n, unsigned per) { return (unsigned)((n + per - 1) / per); }

}  // namespace

namespace {

// How many CTA pairs of the pair kernel the device holds at once (0 = clusters of two cannot be placed).
template <int EPI, bool RESIDENT_W = true>
int ws2_resident_clusters(ullis_cuda_runtime* rt) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // as ullis_cuda_runtime::chain
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(2u * (unsigned)rt->sm_count);
    cfg.blockDim = dim3(WS2_THREADS);
    cfg.dynamicSmemBytes = WS_SMEM_LIMIT;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_ws2_kernel<EPI, RESIDENT_W>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

bool usable(ullis_cuda_runtime* rt) {
    if (rt->mode == ULLIS_CUDA_MODE_EXACT) return false;
    if (rt->tc_ready == 0) {
        rt->tc_ready = -1;
        if (rt->cc_major == 10 && !getenv("ULLIS_CUDA_NO_TC")) {
            encode_fn();
            const int smem = (int)WS_SMEM_LIMIT;
#define ULLIS_SET_SMEM(EPI, PACKED) \
    ULLIS_CUDA_CHECK(cudaFuncSetAttribute(gemm_kernel<EPI, PACKED>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem))
            ULLIS_SET_SMEM(EPI_STORE, true);
            ULLIS_SET_SMEM(EPI_STORE, false);
            ULLIS_SET_SMEM(EPI_RESIDUAL, true);
            ULLIS_SET_SMEM(EPI_RESIDUAL, false);
            ULLIS_SET_SMEM(EPI_RELU2, true);
#define ULLIS_SET_SMEM_NARROW(EPI, PACKED)                                                                                      \
    ULLIS_CUDA_CHECK(cudaFuncSetAttribute(gemm_kernel<EPI, PACKED, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));    \
    ULLIS_CUDA_CHECK(cudaFuncSetAttribute(gemm_kernel<EPI, PACKED, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem))
            ULLIS_SET_SMEM_NARROW(EPI_STORE, true);
            ULLIS_SET_SMEM_NARROW(EPI_STORE, false);
            ULLIS_SET_SMEM_NARROW(EPI_RESIDUAL, true);
            ULLIS_SET_SMEM_NARROW(EPI_RESIDUAL, false);
            ULLIS_SET_SMEM_NARROW(EPI_RELU2, true);
            ULLIS_CUDA_CHECK(cudaFuncSetAttribute(gemm_kernel<EPI_SIGNBITS, true, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
#undef ULLIS_SET_SMEM_NARROW
            ULLIS_SET_SMEM(EPI_SIGNBITS, true);
            ULLIS_SET_SMEM(EPI_CE, true);
#undef ULLIS_SET_SMEM
#define ULLIS_SET_SMEM_WS(EPI) \
    ULLIS_CUDA_CHECK(cudaFuncSetAttribute(gemm_ws_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WS_SMEM_LIMIT))
            ULLIS_SET_SMEM_WS(EPI_STORE);
            ULLIS_SET_SMEM_WS(EPI_RESIDUAL);
            ULLIS_SET_SMEM_WS(EPI_RELU2);
            ULLIS_SET_SMEM_WS(EPI_SIGNBITS);
            ULLIS_SET_SMEM_WS(EPI_CE);
#undef ULLIS_SET_SMEM_WS
            ULLIS_CUDA_CHECK(cudaFuncSetAttribute(gemm_ws_kernel<EPI_STORE, false>,
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WS_SMEM_LIMIT));
            ULLIS_CUDA_CHECK(cudaFuncSetAttribute(gemm_ws_kernel<EPI_RESIDUAL, false>,
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WS_SMEM_LIMIT));
            rt->tc_ws_kernel = !getenv("ULLIS_CUDA_NO_WS");
#define ULLIS_SET_SMEM_WS2(EPI)                                                                                    \
    ULLIS_CUDA_CHECK(cudaFuncSetAttribute(gemm_ws2_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,       \
                                          (int)WS_SMEM_LIMIT));                                                    \
    rt->tc_ws2_clusters[EPI] = ws2_resident_clusters<EPI>(rt)
            ULLIS_SET_SMEM_WS2(EPI_STORE);
            ULLIS_SET_SMEM_WS2(EPI_RESIDUAL);
            ULLIS_SET_SMEM_WS2(EPI_RELU2);
            ULLIS_SET_SMEM_WS2(EPI_SIGNBITS);
            ULLIS_SET_SMEM_WS2(EPI_CE);
#undef ULLIS_SET_SMEM_WS2
            ULLIS_CUDA_CHECK(cudaFuncSetAttribute(gemm_ws2_kernel<EPI_STORE, false>,
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WS_SMEM_LIMIT));
            ULLIS_CUDA_CHECK(cudaFuncSetAttribute(gemm_ws2_kernel<EPI_RESIDUAL, false>,
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WS_SMEM_LIMIT));
            ULLIS_CUDA_CHECK(cudaFuncSetAttribute(gemm_ws2_kernel<EPI_CMIX_GRAD, false>,
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WS_SMEM_LIMIT));
            rt->tc_ws2_dense_clusters[0] = ws2_resident_clusters<EPI_STORE, false>(rt);
            rt->tc_ws2_dense_clusters[1] = ws2_resident_clusters<EPI_RESIDUAL, false>(rt);
            rt->tc_ws2_kernel = rt->tc_ws_kernel && !getenv("ULLIS_CUDA_NO_WS2");
            if (const char* env = getenv("ULLIS_CUDA_WS2_MIN_ROWS")) rt->tc_ws2_min_rows = (size_t)std::max(1, atoi(env));
            ULLIS_CUDA_CHECK(cudaFuncSetAttribute(sign_fixup_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  FIX_QUEUE * 4));
            rt->tc_ready = 1;
        }
    }
    return rt->tc_ready == 1;
}

bool shape_ok(size_t M, size_t K, size_t N) {
    return M > 0 && K >= BK && K % BK == 0 && N >= 8 && N % 8 == 0 && M < (1u << 30) && N < (1u << 30) &&
           (M + BM - 1) / BM <= 65535;
}

// packed weights with a short K go to the weight-stationary kernel
bool takes_ws(const ullis_cuda_runtime* rt, size_t K, uint32_t n_a) {
    return rt->tc_ws_kernel && K / BK <= WS_MAX_KB && ws_shape((uint32_t)K, n_a, true).stages >= 2;
}

// ... and, with enough rows and whole 256-column tiles, to its CTA-pair form
bool takes_ws2(const ullis_cuda_runtime* rt, int epi, size_t M, size_t K, size_t N, uint32_t n_a) {
    return rt->tc_ws2_kernel && takes_ws(rt, K, n_a) && N % WS2_BN == 0 && M >= rt->tc_ws2_min_rows &&
           rt->tc_ws2_clusters[epi] >= 8 && ws2_shape((uint32_t)K, n_a, epi).stages >= 2;
}

// one (problem, 256-column tile) per CTA pair; the pairs with the same one share the 256-row tiles
template <int EPI, bool RESIDENT_W>
void launch_ws2(ullis_cuda_runtime* rt, const GemmMaps& maps, const GemmParams& p, unsigned n_prob, int resident,
                const char* what) {
    const WsShape shape = ws2_shape(p.K, p.n_a, EPI, RESIDENT_W);
    GemmParams q = p;
    q.stages = shape.stages;
    const uint32_t pairs = n_prob * (p.N / WS2_BN) * std::max(p.split_k, 1u), m_tiles = (p.M + WS2_BM - 1) / WS2_BM;
    uint32_t members = (uint32_t)resident / pairs;
    if (members < 1) members = 1;
    if (members > m_tiles) members = m_tiles;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // as ullis_cuda_runtime::chain
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(2u * pairs * members);
    cfg.blockDim = dim3(WS2_THREADS);
    cfg.dynamicSmemBytes = shape.smem;
    cfg.stream = rt->stream;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    if (rt->kernel_timing) rt->mark("(cta_pair)");   // a zero-length entry in the timing table: which form ran
    ULLIS_CUDA_CHECK(cudaLaunchKernelEx(&cfg, gemm_ws2_kernel<EPI, RESIDENT_W>, maps, q, pairs));
    rt->launched(what);
}

// Pipeline depth of gemm_kernel: shallow where three CTAs share an SM (one's epilogue runs under another's MMAs), as deep as
// the shared memory of one or two CTAs allows where the grid leaves no more than that to an SM: a CTA by itself with two
// stages waits for memory at every k-block (K = 2 048, 2 048 rows of 512: 28 -> 25 us).
uint32_t stages_for(const ullis_cuda_runtime* rt, const GemmParams& p, size_t ctas) {
    const size_t per_sm = (ctas + rt->sm_count - 1) / rt->sm_count;
    if (per_sm > 2) return p.stages;
    const size_t room = WS_SMEM_LIMIT / per_sm - 1024 * (per_sm - 1), fixed = gemm_smem_bytes(p.n_a, 0);
    const uint32_t fit = (uint32_t)((room - fixed) / gemm_stage_bytes(p.n_a, p.columns));
    return std::max(p.stages, std::min({fit, (uint32_t)MAX_STAGES, p.K / BK}));
}

// Whether the pair kernel takes dense weights.  It needs half of the pairs at work, or the smaller tiles of gemm_kernel
// spread the rows better (K = 2 048, 16 384 rows of 512, 128 tiles on 74 pairs: 65 -> 43 us; 7 680 rows, 60: 34 -> 31).
template <int EPI>
bool takes_ws2_dense(const ullis_cuda_runtime* rt, const GemmParams& p, unsigned n_prob) {
    const size_t tiles = (size_t)n_prob * ((p.M + WS2_BM - 1) / WS2_BM) * (p.N / WS2_BN);
    const int resident = rt->tc_ws2_dense_clusters[EPI == EPI_RESIDUAL];
    return rt->tc_ws2_kernel && p.N % WS2_BN == 0 && resident >= 8 &&
           2 * tiles * std::max(p.split_k, 1u) >= (size_t)resident &&
           ws2_shape(p.K, p.n_a, EPI, false).stages >= 2;
}

// Columns of gemm_kernel's tiles for M x N outputs: as few as still leave no SM two tiles.  Narrow tiles read the activations more
// often, from L2, but a launch of few rows lasts as long as one CTA: what it brings in (32 KB per k-block with 128 columns, 20 with 32),
// its products and its epilogue.  us of a launch, with the brackets of events: 512 rows, value (K = 1024, 256 columns) 18 -> 14, O (K = 256)
// 14 -> 10, key (1024 columns) 13 -> 10; 2048 rows of 512, value (K = 2048) 25 -> 21, O 17.5 -> 14.  Default model, one sequence 1975 ->
// 1902 us, small model 546 -> 475.
uint32_t tile_columns(const ullis_cuda_runtime* rt, size_t M, size_t N, size_t n_prob = 1) {
    const auto tiles = [&](size_t columns) { return n_prob * ((M + BM - 1) / BM) * ((N + columns - 1) / columns); };
    for (uint32_t columns : {32u, 64u})
        if (tiles(columns) <= (size_t)rt->sm_count) return columns;
    return BN;
}

template <int EPI, bool PACKED>
void launch(ullis_cuda_runtime* rt, const GemmMaps& maps, const GemmParams& p, unsigned n_prob, const char* what) {
    if (PACKED && takes_ws2(rt, EPI, p.M, p.K, p.N, p.n_a)) {
        launch_ws2<EPI, true>(rt, maps, p, n_prob, rt->tc_ws2_clusters[EPI], what);
        return;
    }
    if constexpr (EPI != EPI_CE) {   // its partials are those of 128 columns
        if (p.columns < BN) {
            GemmParams q = p;
            const dim3 grid((p.N + p.columns - 1) / p.columns, (p.M + BM - 1) / BM, n_prob);
            q.stages = stages_for(rt, p, (size_t)grid.x * grid.y * grid.z);
            const size_t smem = gemm_smem_bytes(q.n_a, q.stages, q.columns);
            auto kernel = gemm_kernel<EPI, PACKED, 32>;
            if constexpr (EPI != EPI_SIGNBITS)   // 128 or 32 (rosa_qkv_bits)
                if (p.columns == 64) kernel = gemm_kernel<EPI, PACKED, 64>;
            rt->chain(kernel, grid, GEMM_THREADS, smem, maps, q);
            rt->launched(what);
            return;
        }
    }
    if (PACKED && takes_ws(rt, p.K, p.n_a)) {
        // one (problem, column tile) pair per CTA, the CTAs of a pair share the row tiles
        const WsShape shape = ws_shape(p.K, p.n_a, EPI == EPI_STORE || EPI == EPI_RESIDUAL);
        {
            GemmParams q = p;
            q.stages = shape.stages;
            const uint32_t pairs = n_prob * ((p.N + BN - 1) / BN), m_tiles = (p.M + BM - 1) / BM;
            uint32_t members = (uint32_t)rt->sm_count / pairs;
            if (members < 1) members = 1;
            if (members > m_tiles) members = m_tiles;
            rt->chain(gemm_ws_kernel<EPI>, pairs * members, WS_THREADS, shape.smem, maps, q, pairs);
            rt->launched(what);
            return;
        }
    }
    if constexpr (!PACKED && (EPI == EPI_STORE || EPI == EPI_RESIDUAL)) {
        // dense weights: the persistent kernel with the weight tile in the ring (large M only: a CTA needs
        // several row tiles to amortise its set-up)
        const uint32_t m_tiles = (p.M + BM - 1) / BM, pairs = n_prob * ((p.N + BN - 1) / BN);
        if (p.M >= rt->tc_ws2_min_rows && takes_ws2_dense<EPI>(rt, p, n_prob)) {
            launch_ws2<EPI, false>(rt, maps, p, n_prob, rt->tc_ws2_dense_clusters[EPI], what);
            return;
        }
        if (rt->tc_ws_kernel && m_tiles * pairs >= 4u * (uint32_t)rt->sm_count) {
            const WsShape shape = ws_shape(p.K, p.n_a, true, false);
            GemmParams q = p;
            q.stages = shape.stages;
            uint32_t members = (uint32_t)rt->sm_count / pairs;
            if (members < 1) members = 1;
            if (members > m_tiles) members = m_tiles;
            rt->chain(gemm_ws_kernel<EPI, false>, pairs * members, WS_THREADS, shape.smem, maps, q, pairs);
            rt->launched(what);
            return;
        }
    }
    dim3 grid((p.N + BN - 1) / BN, (p.M + BM - 1) / BM, n_prob);
    GemmParams q = p;
    q.stages = stages_for(rt, p, (size_t)grid.x * grid.y * grid.z);
    rt->chain(gemm_kernel<EPI, PACKED>, grid, GEMM_THREADS, gemm_smem_bytes(q.n_a, q.stages), maps, q);
    rt->launched(what);
}

GemmParams base_params(ullis_cuda_runtime* rt, size_t M, size_t N, size_t K) {
    GemmParams p;
    memset(&p, 0, sizeof(p));
    p.M = (uint32_t)M;
    p.N = (uint32_t)N;
    p.K = (uint32_t)K;
    p.n_a = 1;
    p.stages = rt->tc_stages;   // shallow pipeline, several CTAs per SM: one CTA's epilogue runs under another's MMAs
    p.columns = BN;
    p.status = rt->dev_status;
    return p;
}

// LayerNorm + mixes + 16-bit operands in one kernel when the width allows (a multiple of 128 up to 1024 channels);
// returns false when it does not, and the caller runs the two kernels one after the other.
bool launch_ln_mix_split(ullis_cuda_runtime* rt, const float* x, const LayerNormWeights& ln, float* ln_out,
                         const uint16_t* m0, const uint16_t* m1, const uint16_t* m2, uint16_t* hi0, uint16_t* lo0,
                         uint16_t* hi1, uint16_t* lo1, uint16_t* hi2, uint16_t* lo2, float* s1, size_t rows, size_t time,
                         size_t pitch, size_t d, const char* what) {
    if (!rt->tc_fuse_ln || d % 128 != 0 || d > 1024) return false;
    // Rows per warp: one while the rows are too few to fill the device with warps that take more, and no more than help:
    // us at 512 channels with 1 / 4 / 8, one operand: 4096 rows 9 / 8 / 10, 8192 12.8 / 10.2 / 11.7, 16 384 18 / 14 / 13,
    // 131 072 128 / 88 / 82 (floor 61); Q/K/V: 4096 rows 16 / 18 / 25, 8192 25 / 23 / 26, 131 072 293 / 266 / 274 (floor
    // 205).  Without the loads ahead of the row before, every row's weights in front of its sums and single conversions,
    // 131 072 rows took 131 and 281.
    const uint32_t per_warp = rt->tc_ln_rows > 0 ? (uint32_t)rt->tc_ln_rows : rows < 8192 ? 1 : m1 || rows < 16384 ? 4 : 8;
    const unsigned grid = blocks_for(rows, 8 * per_warp);
#define ULLIS_LN_MIX_FORM(V, SEVERAL, MIXES)                                                                             \
    rt->chain_small(ln_mix_split_kernel<V, SEVERAL, MIXES>, grid, 256, 0, x, ln.weight, ln.bias, ln_out, m0, m1, m2, hi0, \
                    lo0, hi1, lo1, hi2, lo2, s1, (uint32_t)rows, (uint32_t)time, (uint32_t)pitch, per_warp)
#define ULLIS_LN_MIX(V)                                                                \
    do {                                                                               \
        if (per_warp > 1 && m1) ULLIS_LN_MIX_FORM(V, true, 3);                         \
        else if (per_warp > 1) ULLIS_LN_MIX_FORM(V, true, 1);                          \
        else if (m1) ULLIS_LN_MIX_FORM(V, false, 3);                                   \
        else ULLIS_LN_MIX_FORM(V, false, 1);                                           \
    } while (0)
    switch (d / 128) {
        case 1: ULLIS_LN_MIX(1); break;
        case 2: ULLIS_LN_MIX(2); break;
        case 3: ULLIS_LN_MIX(3); break;
        case 4: ULLIS_LN_MIX(4); break;
        case 5: ULLIS_LN_MIX(5); break;
        case 6: ULLIS_LN_MIX(6); break;
        case 7: ULLIS_LN_MIX(7); break;
        default: ULLIS_LN_MIX(8); break;
    }
#undef ULLIS_LN_MIX
#undef ULLIS_LN_MIX_FORM
    rt->launched(what);
    return true;
}

// x [rows, K] f32 -> 16-bit operand
void cast16(ullis_cuda_runtime* rt, const float* x, uint16_t* y, size_t rows, size_t K, bool bf16) {
    const size_t n = rows * K;
    rt->chain(cast16_kernel, blocks_for((n + 3) / 4, 256), 256, 0, x, y, n, bf16 ? 1 : 0, K, rt->dev_status);
    rt->launched("cast16");
}

}  // namespace

CUtensorMap slab_map(const void* ptr, size_t rows, size_t K, unsigned box_rows, unsigned box_slabs) {
    CUtensorMap m;
    cuuint64_t dims[3] = {64, rows, K / 64};
    cuuint64_t strides[2] = {K * 2, 128};
    cuuint32_t box[3] = {64, box_rows, box_slabs};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) fail(ULLIS_CUDA_ERR_CUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
    return m;
}

bool binary_linear(ullis_cuda_runtime* rt, const float* x, const uint32_t* bits, const uint16_t* scale,
                   const uint16_t* bias, float* y, size_t rows, size_t in_features, size_t out_features) {
    if (!usable(rt) || !shape_ok(rows, in_features, out_features) || out_features % 4) return false;
    uint16_t* a = rt->tc_ws[0].as<uint16_t>(rows * in_features);
    cast16(rt, x, a, rows, in_features, false);
    GemmMaps maps;
    memset(&maps, 0, sizeof(maps));
    maps.a[0][0] = make_map(a, rows, in_features, false);
    GemmParams p = base_params(rt, rows, out_features, in_features);
    p.prob[0] = GemmProblem{bits, scale, bias, y, nullptr, nullptr};
    p.columns = tile_columns(rt, rows, out_features);
    launch<EPI_STORE, true>(rt, maps, p, 1, "gemm_packed_store");
    return true;
}

bool fp16_linear(ullis_cuda_runtime* rt, const float* x, const uint16_t* w, float* y, size_t rows,
                 size_t in_features, size_t out_features) {
    if (!usable(rt) || !shape_ok(rows, in_features, out_features)) return false;
    // both operands FP16: the weights as stored (no second rounding), the activations with 11 significant
    // bits; an activation beyond the FP16 range is reported by cast16
    uint16_t* a = rt->tc_ws[0].as<uint16_t>(rows * in_features);
    cast16(rt, x, a, rows, in_features, false);
    GemmMaps maps;
    memset(&maps, 0, sizeof(maps));
    maps.a[0][0] = make_map(a, rows, in_features, false);
    GemmParams p = base_params(rt, rows, out_features, in_features);
    p.columns = tile_columns(rt, rows, out_features);
    maps.b[0] = make_map(w, out_features, in_features, false, p.columns);
    p.prob[0] = GemmProblem{nullptr, nullptr, nullptr, y, nullptr, nullptr};
    launch<EPI_STORE, false>(rt, maps, p, 1, "gemm_dense_store");
    return true;
}

namespace {
// y = sum of the split-K partials, in split order
__global__ void splitk_reduce_kernel(const float* __restrict__ part, float* __restrict__ y, uint32_t splits, size_t n) {
    chain_entry();
    const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= n) return;   // n % 4 == 0 (N % 8 == 0)
    float4 acc = *reinterpret_cast<const float4*>(part + i);
    for (uint32_t s = 1; s < splits; ++s) {
        const float4 v = *reinterpret_cast<const float4*>(part + (size_t)s * n + i);
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    *reinterpret_cast<float4*>(y + i) = acc;
}
}  // namespace

bool dense_nt(ullis_cuda_runtime* rt, const uint16_t* a16, const uint16_t* b16, float* y, size_t M, size_t K,
              size_t N, Partials* partials) {
    if (!usable(rt) || !shape_ok(M, K, N)) return false;
    if (partials) *partials = Partials{y, 1};
    GemmMaps maps;
    memset(&maps, 0, sizeof(maps));
    maps.a[0][0] = make_map(a16, M, K, false);
    maps.b[0] = make_map(b16, N, K, false);
    GemmParams p = base_params(rt, M, N, K);
    p.prob[0] = GemmProblem{nullptr, nullptr, nullptr, y, nullptr, nullptr};
    // A long K under a few output tiles (a weight gradient: K = rows of the batch) is split so that the whole GPU works on
    // it; the partials are then summed in split order.  By CTA pairs where the columns allow (512 x 2 048 of 16 384 rows:
    // 48 -> 37 us).
    const auto reduce = [&](float* part, uint32_t splits) {
        if (partials) {
            *partials = Partials{part, splits};
            return;
        }
        const size_t n = M * N;
        rt->chain(splitk_reduce_kernel, blocks_for((n + 3) / 4, 256), 256, 0, part, y, splits, n);
        rt->launched("splitk_reduce");
    };
    if (N % WS2_BN == 0 && K / BK >= 32) {
        const uint32_t pair_tiles = (uint32_t)((M + WS2_BM - 1) / WS2_BM * (N / WS2_BN)), blocks = (uint32_t)(K / BK);
        uint32_t want = std::min((uint32_t)rt->tc_ws2_dense_clusters[EPI_STORE] / pair_tiles, blocks / 8);
        const uint32_t per = want > 1 ? (blocks + want - 1) / want : blocks, splits = (blocks + per - 1) / per;
        GemmParams q = p;
        q.split_k = splits > 1 ? splits : 0;
        if (takes_ws2_dense<EPI_STORE>(rt, q, 1)) {
            float* part = splits > 1 ? rt->tc_ws[8].as<float>((size_t)splits * M * N) : y;
            q.prob[0].out = part;
            launch_ws2<EPI_STORE, false>(rt, maps, q, 1, rt->tc_ws2_dense_clusters[EPI_STORE],
                                         splits > 1 ? "gemm_dense_nt_splitk" : "gemm_dense_nt");
            if (splits > 1) reduce(part, splits);
            return true;
        }
    }
    const uint32_t tiles = (uint32_t)(((M + BM - 1) / BM) * ((N + BN - 1) / BN)), kb = (uint32_t)(K / BK);
    if (tiles < (uint32_t)rt->sm_count && kb >= 32) {
        uint32_t want = (2u * (uint32_t)rt->sm_count + tiles - 1) / tiles;
        want = std::min(std::min(want, kb / 8), 64u);
        const uint32_t per = (kb + want - 1) / want, splits = (kb + per - 1) / per;
        if (splits > 1) {
            float* part = rt->tc_ws[8].as<float>((size_t)splits * M * N);
            p.split_k = splits;
            p.prob[0].out = part;
            dim3 grid((unsigned)((N + BN - 1) / BN), (unsigned)((M + BM - 1) / BM), splits);
            rt->chain(gemm_kernel<EPI_STORE, false>, grid, GEMM_THREADS, gemm_smem_bytes(p.n_a, p.stages), maps, p);
            rt->launched("gemm_dense_nt_splitk");
            reduce(part, splits);
            return true;
        }
    }
    launch<EPI_STORE, false>(rt, maps, p, 1, "gemm_dense_nt");
    return true;
}

// Bound by the epilogue (14 bytes moved and some 30 operations per element).  16 384 rows, K = 512, N = 2048: the product and
// operands_kernel<true> one after the other 60 + 89 us, together 112 (floor 53, 0.34 GB; without stores and key 63, without the
// arithmetic as well 47).  With too few tiles for the pairs, or fewer rows than they take, the two kernels.
bool cmix_grad_operands(ullis_cuda_runtime* rt, const uint16_t* gy16, const uint16_t* w16, const float* key, const uint16_t* scale,
                        uint16_t* rows_out, uint16_t* grad_t, uint16_t* relu2_t, size_t M, size_t K, size_t N, size_t pitch) {
    if (!usable(rt) || !shape_ok(M, K, N) || M < rt->tc_ws2_min_rows) return false;
    GemmParams p = base_params(rt, M, N, K);
    if (!takes_ws2_dense<EPI_CMIX_GRAD>(rt, p, 1)) return false;
    GemmMaps maps;
    memset(&maps, 0, sizeof(maps));
    maps.a[0][0] = make_map(gy16, M, K, false);
    maps.b[0] = make_map(w16, N, K, false);
    p.prob[0] = GemmProblem{nullptr, scale, nullptr, rows_out, grad_t, key, relu2_t, (uint32_t)pitch};
    launch_ws2<EPI_CMIX_GRAD, false>(rt, maps, p, 1, rt->tc_ws2_dense_clusters[EPI_STORE], "gemm_cmix_grad");
    return true;
}

bool rosa_qkv_bits(ullis_cuda_runtime* rt, const float* ln3_out, const LayerWeights& L, uint32_t* q_sw,
                   uint32_t* k_sw, uint32_t* v_sw, size_t batch, size_t time, size_t d, const float* x_before_ln,
                   float* ln3_write) {
    const size_t rows = batch * time;
    // the GEMM's rows: every sequence padded to whole words of 32 steps, so that a warp of its epilogue holds one word
    const size_t wps = (time + 31) / 32, pitch = 32 * wps, prows = batch * pitch;
    if (!usable(rt) || !shape_ok(prows, d, d)) return false;
    const size_t n = prows * d, sw = batch * d * wps;
    uint16_t* op = rt->tc_ws[1].as<uint16_t>(6 * n);   // q/k/v hi, then q/k/v lo
    float* s1 = rt->tc_ws[2].as<float>(3 * prows);
    uint32_t* flags = rt->tc_ws[3].as<uint32_t>(3 * sw);
    // x_before_ln: ln3 has not run yet - it is folded into the operand kernel, which leaves its output in ln3_write
    // (= ln3_out) for the exact fix-up below
    if (!(x_before_ln && launch_ln_mix_split(rt, x_before_ln, L.ln3, ln3_write, L.x_q, L.x_k, L.x_v, op, op + 3 * n, op + n,
                                             op + 4 * n, op + 2 * n, op + 5 * n, s1, rows, time, pitch, d, "ln_mix_split"))) {
        if (x_before_ln) k::layer_norm(rt, x_before_ln, L.ln3.weight, L.ln3.bias, ln3_write, rows, d, false);
        rt->chain_small(mix_split_kernel, blocks_for(rows, 8), 256, 0, ln3_out, L.x_q, L.x_k, L.x_v, op, op + 3 * n, op + n,
                                                                     op + 4 * n, op + 2 * n, op + 5 * n, s1, rows, time, pitch, d);
        rt->launched("mix_split");
    }
    GemmMaps maps;
    memset(&maps, 0, sizeof(maps));
    for (int z = 0; z < 3; ++z) {
        maps.a[z][0] = make_map(op + z * n, prows, d, false);
        maps.a[z][1] = make_map(op + (3 + z) * n, prows, d, false);
    }
    GemmParams p = base_params(rt, prows, d, d);
    p.n_a = 2;
    p.stages = rt->tc_stages2;
    p.time = (uint32_t)pitch;
    p.steps = (uint32_t)time;
    p.wps = (uint32_t)wps;
    const PackedWeights* W[3] = {&L.q, &L.k, &L.v};
    uint32_t* outs[3] = {q_sw, k_sw, v_sw};
    for (int z = 0; z < 3; ++z)
        p.prob[z] = GemmProblem{W[z]->bits, W[z]->scale, W[z]->bias, outs[z], flags + z * sw, s1 + z * prows};
    // 64 columns no better than the kernel that keeps its weights (small model, 3 times 333 steps 457 us, so 444)
    p.columns = tile_columns(rt, prows, d, 3) == 32 ? 32 : BN;
    launch<EPI_SIGNBITS, true>(rt, maps, p, 3, "gemm_qkv_signbits");
    // rows < 2^30, so both grids fit
    if (rt->tc_fix_blocks && fix_block_threads(d) <= FIXB_MAX_THREADS) {   // d % 64 == 0 (shape_ok)
        // A part of a block for each CTA while that makes no more than the device holds at once: with few blocks the chain of one
        // CTA is what lasts, with many the rows that are read twice count.  us of a whole call with 32 / 16 / 8 / 4 steps, 64 blocks:
        // 2 359 / 2 252 / 2 198 / 2 183, 240: 3 928 / 3 672 / 3 607 / 3 703, 512: 6 581 / 6 334 / 6 424 / 6 650, 1024: 8 076 /
        // 8 143 / 8 339 / 8 803.
        const size_t blocks = wps * batch;
        uint32_t steps = 4;
        while (steps < 32 && blocks * (32 / steps) > 8 * (size_t)rt->sm_count) steps *= 2;
        rt->chain(fix_block_kernel, (unsigned)(blocks * (32 / steps)), fix_block_threads(d), fix_block_smem(d), ln3_out, L.x_q, L.x_k,
                  L.x_v, L.q, L.k, L.v, q_sw, k_sw, v_sw, flags, sw, (uint32_t)time, (uint32_t)d, (uint32_t)wps, steps);
        rt->launched("fix_block");
    } else {
        rt->chain(sign_fixup_kernel, (unsigned)(((wps + FIX_WIN - 1) / FIX_WIN) * batch), FIX_THREADS, FIX_QUEUE * 4, ln3_out, L.x_q,
                  L.x_k, L.x_v, L.q, L.k, L.v, q_sw, k_sw, v_sw, flags, flags + sw, flags + 2 * sw, batch, time, d, wps);
        rt->launched("sign_fixup");
    }
    return true;
}

bool rosa_out_residual(ullis_cuda_runtime* rt, const uint32_t* idx_sw, const LayerWeights& L, float* x, size_t batch,
                       size_t time, size_t d) {
    const size_t rows = batch * time;
    if (!usable(rt) || !shape_ok(rows, d, d) || d % 4) return false;
    uint16_t* y16 = rt->tc_ws[0].as<uint16_t>(rows * d);
    const size_t wps = (time + 31) / 32;
    dim3 grid((unsigned)wps, (unsigned)((d + 255) / 256), (unsigned)batch);
    rt->chain(emit_f16_kernel, grid, 256, 0, idx_sw, L.e, y16, time, d, wps);
    rt->launched("emit_f16");
    GemmMaps maps;
    memset(&maps, 0, sizeof(maps));
    maps.a[0][0] = make_map(y16, rows, d, false);
    GemmParams p = base_params(rt, rows, d, d);
    p.prob[0] = GemmProblem{L.o.bits, L.o.scale, L.o.bias, x, nullptr, nullptr};
    p.columns = tile_columns(rt, rows, d);
    launch<EPI_RESIDUAL, true>(rt, maps, p, 1, "gemm_o_residual");
    return true;
}

bool cmix_residual(ullis_cuda_runtime* rt, const LayerWeights& L, float* x, size_t batch, size_t time, size_t d,
                   size_t ffn) {
    const size_t rows = batch * time;
    if (!usable(rt) || !shape_ok(rows, d, ffn) || !shape_ok(rows, ffn, d) || d % 4) return false;
    float* ln = rt->tc_ws[4].as<float>(rows * d);
    uint16_t* a16 = rt->tc_ws[0].as<uint16_t>(rows * d);
    uint16_t* k16 = rt->tc_ws[5].as<uint16_t>(rows * ffn);
    if (!launch_ln_mix_split(rt, x, L.ln2, nullptr, L.ffn_x_k, nullptr, nullptr, a16, nullptr, nullptr, nullptr, nullptr,
                             nullptr, nullptr, rows, time, time, d, "ln_mix_f16")) {
        k::layer_norm(rt, x, L.ln2.weight, L.ln2.bias, ln, rows, d, false);
        rt->chain_small(mix_split_kernel, blocks_for(rows, 8), 256, 0, ln, L.ffn_x_k, nullptr, nullptr, a16, nullptr,
                                                                     nullptr, nullptr, nullptr, nullptr, nullptr, rows, time, time, d);
        rt->launched("mix_f16");
    }
    GemmMaps maps;
    memset(&maps, 0, sizeof(maps));
    maps.a[0][0] = make_map(a16, rows, d, false);
    GemmParams p = base_params(rt, rows, ffn, d);
    p.out_fmt = 0;  // FP16: three more significant bits than bf16; the epilogue reports values past 65504
    p.prob[0] = GemmProblem{L.key.bits, L.key.scale, nullptr, k16, nullptr, nullptr};
    p.columns = tile_columns(rt, rows, ffn);
    launch<EPI_RELU2, true>(rt, maps, p, 1, "gemm_key_relu2");
    memset(&maps, 0, sizeof(maps));
    maps.a[0][0] = make_map(k16, rows, ffn, false);
    GemmParams pv = base_params(rt, rows, d, ffn);
    pv.columns = tile_columns(rt, rows, d);
    maps.b[0] = make_map(L.value, d, ffn, false, pv.columns);   // the FP16 weights as stored
    pv.prob[0] = GemmProblem{nullptr, nullptr, nullptr, x, nullptr, nullptr};
    launch<EPI_RESIDUAL, false>(rt, maps, pv, 1, "gemm_value_residual");
    return true;
}

namespace {
// One CTA waits, with the bounded mbarrier wait every tensor-core kernel here uses, on a barrier that nothing
// ever arrives on, and reports the give-up through the runtime's status words like those kernels do.
__global__ void wait_selftest_kernel(uint32_t polls, uint32_t* status) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        ptx::mbar_init(&bar, 1);
        ptx::fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0 && !ptx::mbar_wait(&bar, 0, polls)) {
        if (atomicCAS(status, ULLIS_DEV_OK, ULLIS_DEV_WAIT_TIMEOUT) == ULLIS_DEV_OK) status[1] = 99u;   // site: self-test
    }
}
}  // namespace

void wait_selftest(ullis_cuda_runtime* rt, uint32_t polls) {
    wait_selftest_kernel<<<1, 32, 0, rt->stream>>>(polls, rt->dev_status);
    rt->launched("wait_selftest");
}

bool takes_model(ullis_cuda_runtime* rt, size_t rows, size_t time, size_t d, size_t ffn, size_t vocab) {
    return usable(rt) && shape_ok((rows + time - 1) / time * ((time + 31) / 32 * 32), d, d) && d % 4 == 0 && shape_ok(rows, d, ffn) &&
           shape_ok(rows, ffn, d) && shape_ok(rows, d, vocab);
}

bool head_ce(ullis_cuda_runtime* rt, const float* hidden, const PackedWeights& head, const uint32_t* labels,
             uint32_t ignore_id, size_t rows, size_t time, size_t d, size_t vocab, float* row_loss) {
    if (!usable(rt) || !shape_ok(rows, d, vocab)) return false;
    // partials per row: one per vocabulary tile and epilogue warp group of the kernel that will run
    const uint32_t n_tiles = (uint32_t)((vocab + BN - 1) / BN) * (takes_ws(rt, d, 1) ? WS_EPI_GROUPS : 1u);
    uint16_t* a16 = rt->tc_ws[0].as<uint16_t>(rows * d);
    float2* part = rt->tc_ws[6].as<float2>(rows * n_tiles);
    float* tl = rt->tc_ws[7].as<float>(rows);
    cast16(rt, hidden, a16, rows, d, false);
    GemmMaps maps;
    memset(&maps, 0, sizeof(maps));
    maps.a[0][0] = make_map(a16, rows, d, false);
    GemmParams p = base_params(rt, rows, vocab, d);
    p.labels = labels;
    p.ignore_id = ignore_id;
    p.n_tiles = n_tiles;
    p.time = (uint32_t)time;
    p.prob[0] = GemmProblem{head.bits, head.scale, head.bias, part, tl, nullptr};
    launch<EPI_CE, true>(rt, maps, p, 1, "gemm_head_ce");
    rt->chain(ce_finish_kernel, blocks_for(rows, 8), 256, 0, part, tl, labels, ignore_id, rows, time, vocab, n_tiles,
                                                                  row_loss, rt->dev_status);
    rt->launched("ce_finish");
    return true;
}

}  // namespace tc
}  // namespace ullis
