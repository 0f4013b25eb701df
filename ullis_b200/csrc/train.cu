// One training step on the device, rosa_grad = stop_grad_bits: the tensor-core
// forward keeps a small tape (the residual stream after each ROSA block and
// the idx bits), the backward recomputes the CMix activations from it and
// runs every gradient matrix product as an FP16 x FP16 -> f32 tcgen05 GEMM on
// operands that small kernels cast / transpose, and the optimiser kernels
// apply the reference's clipped SGD and BinaryConnect steps element by element.
//
// Reference: train_step_on (src/model.rs:2827-3020), apply_head_ce
// (3132-3275), backward_ste (745-796), flip_after_gradients (838-876),
// CMix backward_update (1138-1177), backward_stop_grad (1494-1521),
// rosa_e_grad (1608-1634), LayerNorm::backward (270-315),
// Fp16Storage::apply_clipped_sgd / apply_binaryconnect_sgd (src/precision.rs:106-134).
//
// Gradients travel multiplied by P = 2^ceil(log2(T-1)): the loss scale is
// 1/(T-1), so P*g is O(1) where the 16-bit GEMM operands are formed, and the
// optimiser kernels multiply by 1/P (exact) before they clip.
#include "train.hpp"

#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "kernels.hpp"
#include "linear_tc.hpp"
#include "safetensors.hpp"

using namespace ullis;

namespace {

constexpr float LN_EPS = 1e-5f;              // src/model.rs:22
constexpr float HEAD_BIAS_LR_MULT = 8.0f;    // src/model.rs:97
constexpr uint16_t LATENT_PLUS = 0x211F;     // FP16(0.01), BINARYCONNECT_INIT_ABS (src/model.rs:550)

__device__ __forceinline__ float h2f(uint16_t b) { return __half2float(__ushort_as_half(b)); }

// f32 -> FP16 bits; a finite value beyond the FP16 range is reported, not turned into inf
__device__ __forceinline__ uint16_t to_f16(float v, uint32_t* status, size_t row) {
    const float a = fabsf(v);
    if (a > 65504.0f && a <= 3.4028234e38f) {
        if (atomicCAS(status, ULLIS_DEV_OK, ULLIS_DEV_FP16_RANGE) == ULLIS_DEV_OK) status[1] = (uint32_t)row;
        v = copysignf(65504.0f, v);
    }
    return __half_as_ushort(__float2half_rn(v));
}

inline unsigned blocks_for(size_t n, unsigned per) { return (unsigned)((n + per - 1) / per); }
inline size_t pad64(size_t n) { return (n + 63) / 64 * 64; }

// ------------------------------------------------------------ GEMM operands
// FP16 operands of the gradient products from x [R, C], both ways in one pass over it:
//   rows_out [R, Cp] = FP16(x * colscale[c]), columns C..Cp zero (null: not wanted)
//   t_out    [C, Rp] = FP16(x)^T, columns R..Rp zero
// CMIX: x is g_relu2 and `key` the pre-activation; x becomes g_key = key > 0 ? 2 * key * x : 0 (relu2_bwd_on,
// src/model.rs:1189-1204) first, and relu2_t [C, Rp] = FP16(relu(key)^2)^T leaves as well.
// Bound by memory: a CTA moves 64 rows x 64 columns, 16-byte loads along a row, 16-byte stores of eight rows of a column.
// As relu^2 backward, cast and two transposes one after the other the CMix part moved 1.0 GB per layer at 16 384 rows of
// 2 048, in one pass 0.47 GB.
template <bool CMIX>
__global__ void __launch_bounds__(256)
operands_kernel(const float* __restrict__ x, const float* __restrict__ key, const uint16_t* __restrict__ colscale,
                uint16_t* __restrict__ rows_out, uint16_t* __restrict__ t_out, uint16_t* __restrict__ relu2_t, size_t R,
                size_t C, size_t Cp, size_t Rp, uint32_t* status) {
    chain_entry();
    __shared__ uint16_t tile[CMIX ? 2 : 1][64][66];
    const size_t r0 = (size_t)blockIdx.x * 64, c0 = (size_t)blockIdx.y * 64;
    const bool vec = (C & 3) == 0;
    const auto load = [&](const float* from, size_t r, size_t c, float* v) {
        if (vec && c + 3 < C) {
            const float4 t = *reinterpret_cast<const float4*>(from + r * C + c);
            v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
        } else {
            for (int e = 0; e < 4; ++e) v[e] = c + e < C ? from[r * C + c + e] : 0.0f;
        }
    };
    float v[4][4] = {}, kv[CMIX ? 4 : 1][4] = {};
#pragma unroll
    for (int k = 0; k < 4; ++k) {   // 64 rows x 16 groups of four columns
        const size_t r = r0 + ((threadIdx.x + k * 256) >> 4), c = c0 + (threadIdx.x & 15) * 4;
        if (r < R) load(x, r, c, v[k]);
        if (CMIX && r < R) load(key, r, c, kv[CMIX ? k : 0]);
    }
    const int q = (threadIdx.x & 15) * 4;
    float scale[4] = {1.0f, 1.0f, 1.0f, 1.0f};
    if (rows_out && colscale)
        for (int e = 0; e < 4; ++e) if (c0 + q + e < C) scale[e] = h2f(colscale[c0 + q + e]);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int j = (threadIdx.x + k * 256) >> 4;
        uint16_t row[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float t = v[k][e];
            if (CMIX) {
                const float y = kv[CMIX ? k : 0][e];
                t = y > 0.0f ? 2.0f * y * t : 0.0f;
                const float relu = fmaxf(y, 0.0f);
                tile[CMIX ? 1 : 0][j][q + e] = to_f16(relu * relu, status, r0 + j);
            }
            tile[0][j][q + e] = to_f16(t, status, r0 + j);
            row[e] = to_f16(colscale ? __fmul_rn(t, scale[e]) : t, status, r0 + j);
        }
        if (rows_out && r0 + j < R)
            *reinterpret_cast<uint2*>(rows_out + (r0 + j) * Cp + c0 + q) =
                make_uint2(row[0] | (uint32_t)row[1] << 16, row[2] | (uint32_t)row[3] << 16);
    }
    __syncthreads();
    const int cl = threadIdx.x >> 2, seg = (threadIdx.x & 3) * 16;   // column, first of its sixteen rows
    const size_t c = c0 + cl;
    if (c >= C) return;
#pragma unroll
    for (int which = 0; which < (CMIX ? 2 : 1); ++which) {
        uint16_t* out = which ? relu2_t : t_out;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int j = seg + h * 8 + e * 2;
                w[e] = tile[which][j][cl] | (uint32_t)tile[which][j + 1][cl] << 16;
            }
            // r0 + seg + 8h + 7 < Rp: Rp is a multiple of 64
            *reinterpret_cast<uint4*>(out + c * Rp + r0 + seg + h * 8) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

// packed signs [out, in] -> FP16 +/-1 [in, outp], columns out..outp zero
__global__ void unpack_transpose_kernel(const uint32_t* __restrict__ bits, uint16_t* __restrict__ b16, size_t out_f,
                                        size_t in_f, size_t outp) {
    chain_entry();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= in_f * outp) return;
    const size_t k = i / outp, o = i % outp;
    uint16_t v = 0;
    if (o < out_f) {
        const size_t bit = o * in_f + k;
        v = (bits[bit >> 5] >> (bit & 31)) & 1u ? 0x3C00 : 0xBC00;
    }
    b16[i] = v;
}

// w [R, C] FP16 -> [C, Rp], columns R..Rp zero; a CTA has 64 rows x 64 columns
__global__ void __launch_bounds__(256)
transpose16_kernel(const uint16_t* __restrict__ w, uint16_t* __restrict__ out, size_t R, size_t C, size_t Rp) {
    chain_entry();
    __shared__ uint16_t tile[64][66];
    const size_t r0 = (size_t)blockIdx.x * 64, c0 = (size_t)blockIdx.y * 64;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const int j = (threadIdx.x >> 6) + k * 4, q = threadIdx.x & 63;
        tile[j][q] = r0 + j < R && c0 + q < C ? w[(r0 + j) * C + c0 + q] : (uint16_t)0;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const int j = threadIdx.x & 63, q = (threadIdx.x >> 6) + k * 4;
        if (c0 + q < C) out[(c0 + q) * Rp + r0 + j] = tile[j][q];   // r0 + j < Rp: Rp is a multiple of 64
    }
}

// y [M, N] = a [M, K] . b [N, K]^T, f32 accumulation of the same FP16 operands the
// tensor-core kernel takes (shapes outside its tiling, validation mode)
__global__ void gemm_nt_plain_kernel(const uint16_t* __restrict__ a, const uint16_t* __restrict__ b,
                                     float* __restrict__ y, size_t M, size_t K, size_t N) {
    __shared__ float sa[16][17], sb[16][17];
    const size_t m = (size_t)blockIdx.y * 16 + threadIdx.y, n = (size_t)blockIdx.x * 16 + threadIdx.x;
    float acc = 0.0f;
    for (size_t k0 = 0; k0 < K; k0 += 16) {
        const size_t ka = k0 + threadIdx.x;
        sa[threadIdx.y][threadIdx.x] = (m < M && ka < K) ? h2f(a[m * K + ka]) : 0.0f;
        const size_t nb = (size_t)blockIdx.x * 16 + threadIdx.y;
        sb[threadIdx.y][threadIdx.x] = (nb < N && ka < K) ? h2f(b[nb * K + ka]) : 0.0f;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; ++k) acc = fmaf(sa[threadIdx.y][k], sb[threadIdx.x][k], acc);
        __syncthreads();
    }
    if (m < M && n < N) y[m * N + n] = acc;
}

// ------------------------------------------------------------ head
// logits [rows, V] -> row_loss and, in place, gy * P with gy = loss_scale * (softmax - onehot)
// (src/model.rs:3204-3236; valid-row rule 27-39).  One CTA per row.
__global__ void __launch_bounds__(256)
ce_grad_kernel(float* __restrict__ logits, const uint32_t* __restrict__ labels, uint32_t ignore_id, size_t rows,
               size_t time, size_t vocab, float loss_scale, float P, float* __restrict__ row_loss,
               uint32_t* status) {
    chain_entry();
    __shared__ float red[8];
    __shared__ float bcast;
    const size_t m = blockIdx.x;
    float* lg = logits + m * vocab;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    bool valid = (m % time) + 1 < time && m + 1 < rows && labels[m + 1] != ignore_id;
    const uint32_t target = valid ? labels[m + 1] : 0u;
    if (valid && target >= vocab) {
        if (threadIdx.x == 0 && atomicCAS(status, ULLIS_DEV_OK, ULLIS_DEV_BAD_TOKEN) == ULLIS_DEV_OK)
            status[1] = (uint32_t)m;
        valid = false;
    }
    if (!valid) {
        for (size_t v = threadIdx.x; v < vocab; v += 256) lg[v] = 0.0f;
        if (threadIdx.x == 0) row_loss[m] = 0.0f;
        return;
    }
    float mx = -INFINITY;
    for (size_t v = threadIdx.x; v < vocab; v += 256) mx = fmaxf(mx, lg[v]);
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) red[warp] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        float v = red[0];
        for (int w = 1; w < 8; ++w) v = fmaxf(v, red[w]);
        bcast = v;
    }
    __syncthreads();
    mx = bcast;
    float sum = 0.0f;
    for (size_t v = threadIdx.x; v < vocab; v += 256) sum += expf(lg[v] - mx);
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    __syncthreads();
    if (lane == 0) red[warp] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        float v = 0.0f;
        for (int w = 0; w < 8; ++w) v += red[w];
        bcast = v;
        row_loss[m] = mx + logf(v) - lg[target];
    }
    __syncthreads();
    sum = bcast;
    for (size_t v = threadIdx.x; v < vocab; v += 256) {
        const float p = expf(lg[v] - mx) / sum;
        lg[v] = loss_scale * (p - (v == target ? 1.0f : 0.0f)) * P;
    }
}

// ------------------------------------------------------------ reductions over rows
// part[chunk, c] = sum over the chunk's 256 rows of f(a, b):
//   COL_SUM    a
//   COL_LN     a * (b - mean) / deviation, by the row's statistics, and a in a second part behind the first
//   COL_SHIFT  a * (b of the row before - b), 0 before the first row of a sequence
//   COL_SIGN   b ? a : -a                                   b u8 [R, C]
//   COL_BITS   the same, b stream-major bits
// Bound by bringing the rows in: a warp has 16 rows of 32 columns on their way at a time, a column per lane, and adds up its own; the
// eight sums of a CTA meet in shared memory.  (With the rows in shared memory and one warp that adds up 128 of them the chain was
// what lasted: the 102 sums of two steps of 8 x 2048 tokens 2.23 ms between events, now 2.07.)
enum ColMode { COL_SUM, COL_LN, COL_SHIFT, COL_SIGN, COL_BITS };
constexpr int COL_ROWS = 256, COL_STEP = 128, COL_WARP_ROWS = COL_STEP / 8;
template <ColMode MODE>
__global__ void __launch_bounds__(256)
col_partial_kernel(const float* __restrict__ a, const void* __restrict__ b, const float2* __restrict__ stats,
                   float* __restrict__ part, uint32_t R, uint32_t C, uint32_t time) {
    chain_entry();
    constexpr bool PRODUCT = MODE == COL_LN || MODE == COL_SHIFT;
    __shared__ float sums[2][8][32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, c = blockIdx.x * 32u + lane;
    const uint32_t r0 = blockIdx.y * COL_ROWS, r1 = min(r0 + COL_ROWS, R);
    const float* b32 = static_cast<const float*>(b);
    float acc = 0.0f, plain = 0.0f;
    for (uint32_t h = r0; h < r1; h += COL_STEP) {
        const uint32_t rw = h + warp * COL_WARP_ROWS;
        float av[COL_WARP_ROWS] = {}, bv[COL_WARP_ROWS] = {};
        if (c < C) {
            if (rw + COL_WARP_ROWS <= r1) {
#pragma unroll
                for (int i = 0; i < COL_WARP_ROWS; ++i) {
                    av[i] = a[(size_t)(rw + i) * C + c];
                    if (PRODUCT) bv[i] = b32[(size_t)(rw + i) * C + c];
                    if (MODE == COL_SIGN) bv[i] = static_cast<const uint8_t*>(b)[(size_t)(rw + i) * C + c];
                }
            } else {
#pragma unroll
                for (int i = 0; i < COL_WARP_ROWS; ++i)
                    if (rw + i < r1) {
                        av[i] = a[(size_t)(rw + i) * C + c];
                        if (PRODUCT) bv[i] = b32[(size_t)(rw + i) * C + c];
                        if (MODE == COL_SIGN) bv[i] = static_cast<const uint8_t*>(b)[(size_t)(rw + i) * C + c];
                    }
            }
            if (MODE == COL_LN) {
#pragma unroll
                for (int i = 0; i < COL_WARP_ROWS; ++i)
                    if (rw + i < r1) {
                        const float2 st = stats[rw + i];
                        bv[i] = (bv[i] - st.x) * st.y;
                    }
            }
            if (MODE == COL_SHIFT && rw < r1) {
                uint32_t t = rw % time;
                float before = t ? b32[(size_t)(rw - 1) * C + c] : 0.0f;
#pragma unroll
                for (int i = 0; i < COL_WARP_ROWS; ++i) {
                    const float now = bv[i];
                    bv[i] = t ? __fsub_rn(before, now) : -now;
                    before = now;
                    t = t + 1 == time ? 0 : t + 1;
                }
            }
            if (MODE == COL_BITS && rw < r1) {
                const uint32_t wps = (time + 31u) / 32u;
                uint32_t seq = rw / time, t = rw - seq * time, word = 0;
                for (int i = 0; i < COL_WARP_ROWS; ++i) {
                    if (i == 0 || (t & 31u) == 0u)
                        word = rw + i < r1 ? static_cast<const uint32_t*>(b)[((size_t)seq * C + c) * wps + (t >> 5)] : 0u;
                    bv[i] = (float)((word >> (t & 31u)) & 1u);
                    if (++t == time) { t = 0; ++seq; }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < COL_WARP_ROWS; ++i) {   // rows past the last are zeros
            if (PRODUCT) acc += av[i] * bv[i];
            else acc += (MODE == COL_SIGN || MODE == COL_BITS) && bv[i] == 0.0f ? -av[i] : av[i];
            if (MODE == COL_LN) plain += av[i];
        }
    }
    sums[0][warp][lane] = acc;
    if (MODE == COL_LN) sums[1][warp][lane] = plain;
    __syncthreads();
    if (c < C && warp < (MODE == COL_LN ? 2u : 1u)) {
        float all = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; ++w) all += sums[warp][w][lane];
        part[((size_t)warp * gridDim.y + blockIdx.y) * C + c] = all;
    }
}

// Fp16Storage::apply_clipped_sgd (src/precision.rs:106-113) on g * gmul
__device__ __forceinline__ void clipped_step(uint16_t& w, float& residual, float g, float lr) {
    const float current = h2f(w);
    const float update = __fmul_rn(lr, fminf(fmaxf(g, -1.0f), 1.0f));
    const float desired = __fadd_rn(__fsub_rn(current, update), residual);
    const uint16_t rounded = __half_as_ushort(__float2half_rn(desired));
    residual = __fsub_rn(desired, h2f(rounded));
    w = rounded;
}

// FP16 parameters that a column sum (or two) is the gradient of; null: the sums themselves are wanted.
struct ColStep {
    uint16_t* w[2];
    float* residual[2];
    float gmul, lr;
};

// out[y, c] = sum over the chunks of part[y, chunk, c]; or the step that it is the gradient for, at once (as a launch of its own each of
// these vectors of 512 took a training step 2.5 us, 62 of them).
__global__ void __launch_bounds__(64)
col_final_kernel(const float* __restrict__ part, float* __restrict__ out, size_t chunks, size_t C, const ColStep step) {
    chain_entry();
    const size_t c = (size_t)blockIdx.x * 64 + threadIdx.x;
    if (c >= C) return;
    part += blockIdx.y * chunks * C + c;
    float acc = 0.0f;
    size_t k = 0;
    for (; k + 16 <= chunks; k += 16) {
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = part[(k + i) * C];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc += v[i];
    }
    for (; k < chunks; ++k) acc += part[k * C];
    if (step.w[0]) clipped_step(step.w[blockIdx.y][c], step.residual[blockIdx.y][c], __fmul_rn(acc, step.gmul), step.lr);
    else out[blockIdx.y * C + c] = acc;
}

// ------------------------------------------------------------ LayerNorm backward
// gx (+)= d/dx, and the row's mean and 1 / deviation (for g_w = sum gy * xhat); one warp per row (src/model.rs:270-315).
// N > 0: C = 32 * N, the row, its gradient and the old gx in registers (all loads in flight together, each read once); N = 0:
// any C, the same sums in the same order.  16 384 rows of 512 added to gx: 47 -> 20 us (an f32 row per column sum was
// written besides before).
template <int N>
__global__ void __launch_bounds__(256)
ln_backward_kernel(const float* __restrict__ x, const float* __restrict__ gy, const uint16_t* __restrict__ w,
                   float* __restrict__ gx, float2* __restrict__ stats, size_t rows, size_t C, int accumulate) {
    chain_entry();
    const int lane = threadIdx.x & 31;
    const size_t row = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    const float* xr = x + row * C;
    const float* gr = gy + row * C;
    float xs[N ? N : 1], gs[N ? N : 1], old[N ? N : 1];
    if constexpr (N > 0) {
#pragma unroll
        for (int i = 0; i < N; ++i) xs[i] = xr[lane + 32 * i];
#pragma unroll
        for (int i = 0; i < N; ++i) gs[i] = gr[lane + 32 * i];
#pragma unroll
        for (int i = 0; i < N; ++i) old[i] = accumulate ? gx[row * C + lane + 32 * i] : 0.0f;
    }
    const auto each = [&](auto f) {   // f(column, x, gy)
        if constexpr (N > 0) {
#pragma unroll
            for (int i = 0; i < N; ++i) f((size_t)(lane + 32 * i), xs[i], gs[i]);
        } else {
            for (size_t c = lane; c < C; c += 32) f(c, xr[c], gr[c]);
        }
    };
    float s = 0.0f;
    each([&](size_t, float xv, float) { s += xv; });
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float mean = s / (float)C;
    float v = 0.0f;
    each([&](size_t, float xv, float) { const float dlt = xv - mean; v += dlt * dlt; });
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const float inv = 1.0f / sqrtf(v / (float)C + LN_EPS);
    float s1 = 0.0f, s2 = 0.0f;
    each([&](size_t c, float xv, float gv) {
        const float xh = (xv - mean) * inv, dx = gv * h2f(w[c]);
        s1 += dx;
        s2 += dx * xh;
    });
    for (int o = 16; o > 0; o >>= 1) {
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    const float inv_n = inv / (float)C;
    if (lane == 0) stats[row] = make_float2(mean, inv);
    if constexpr (N > 0) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const float xh = (xs[i] - mean) * inv, dx = gs[i] * h2f(w[lane + 32 * i]);
            const float g = inv_n * ((float)C * dx - s1 - xh * s2);
            gx[row * C + lane + 32 * i] = accumulate ? old[i] + g : g;
        }
    } else {
        for (size_t c = lane; c < C; c += 32) {
            const float xh = (xr[c] - mean) * inv, dx = gr[c] * h2f(w[c]);
            const float g = inv_n * ((float)C * dx - s1 - xh * s2);
            gx[row * C + c] = accumulate ? gx[row * C + c] + g : g;
        }
    }
}

// Widths of up to 1024 that a warp can take into registers whole, in steps of 32 up to 128 and of 128 above (as far as
// LayerNorm goes forward); the others loop over the row.  us for 16 384 rows, loop / registers: 64 columns 12.0 / 6.3, 128
// 12.1 / 8.0, 256 17.7 / 10.3, 384 23.0 / 13.6, 512 31.3 / 17.0, 640 37.2 / 23.3, 768 45.7 / 25.0, 896 52.5 / 28.2, 1024
// 64.4 / 31.9; for 1000 rows 5.4 / 3.6 to 23.7 / 5.4.
void ln_backward_launch(ullis_cuda_runtime* rt, const float* x, const float* gy, const uint16_t* w, float* gx, float2* stats,
                        size_t rows, size_t C, int accumulate) {
    const unsigned grid = blocks_for(rows, 8);
    switch (C % 32 == 0 ? C / 32 : 0) {
#define ULLIS_LN_BACKWARD(N) \
    case N: rt->chain(ln_backward_kernel<N>, grid, 256, 0, x, gy, w, gx, stats, rows, C, accumulate); break
        ULLIS_LN_BACKWARD(1); ULLIS_LN_BACKWARD(2); ULLIS_LN_BACKWARD(3); ULLIS_LN_BACKWARD(4);
        ULLIS_LN_BACKWARD(8); ULLIS_LN_BACKWARD(12); ULLIS_LN_BACKWARD(16); ULLIS_LN_BACKWARD(20);
        ULLIS_LN_BACKWARD(24); ULLIS_LN_BACKWARD(28); ULLIS_LN_BACKWARD(32);
#undef ULLIS_LN_BACKWARD
        default: rt->chain(ln_backward_kernel<0>, grid, 256, 0, x, gy, w, gx, stats, rows, C, accumulate);
    }
    rt->launched("ln_backward");
}

// ------------------------------------------------------------ CMix pieces
// g <- key > 0 ? 2*key*g : 0   (relu2_bwd_on, src/model.rs:1189-1204)
__global__ void relu2_bwd_kernel(const float* __restrict__ key, float* __restrict__ g, size_t n) {
    chain_entry();
    const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= n) return;
    if (i + 4 <= n) {
        const float4 k = *reinterpret_cast<const float4*>(key + i);
        float4 v = *reinterpret_cast<const float4*>(g + i);
        v.x = k.x > 0.0f ? 2.0f * k.x * v.x : 0.0f;
        v.y = k.y > 0.0f ? 2.0f * k.y * v.y : 0.0f;
        v.z = k.z > 0.0f ? 2.0f * k.z * v.z : 0.0f;
        v.w = k.w > 0.0f ? 2.0f * k.w * v.w : 0.0f;
        *reinterpret_cast<float4*>(g + i) = v;
        return;
    }
    for (size_t j = i; j < n; ++j) g[j] = key[j] > 0.0f ? 2.0f * key[j] * g[j] : 0.0f;
}

// lerp_shift_backward (src/model.rs:1206-1240): out[t] = (g[t] - g[t]*mix) + g[t+1]*mix.  Four columns per thread
// (C % 4 == 0), or one.
template <int N>
__global__ void lerp_bwd_kernel(const float* __restrict__ g, const uint16_t* __restrict__ mix, float* __restrict__ out,
                                uint32_t rows, uint32_t time, uint32_t C) {
    chain_entry();
    const uint32_t per_row = C / N, i = blockIdx.x * blockDim.x + threadIdx.x, row = i / per_row;
    if (row >= rows) return;
    const uint32_t c = (i - row * per_row) * N;
    const size_t at = (size_t)row * C + c;
    const bool more = row % time + 1u < time;
    float now[N], next[N], res[N];
    if constexpr (N == 4) {
        const float4 a = *reinterpret_cast<const float4*>(g + at), b = more ? *reinterpret_cast<const float4*>(g + at + C) : a;
        now[0] = a.x; now[1] = a.y; now[2] = a.z; now[3] = a.w;
        next[0] = b.x; next[1] = b.y; next[2] = b.z; next[3] = b.w;
    } else {
        now[0] = g[at];
        next[0] = more ? g[at + C] : 0.0f;
    }
#pragma unroll
    for (int e = 0; e < N; ++e) {
        const float mv = h2f(mix[c + e]);
        res[e] = __fsub_rn(now[e], __fmul_rn(now[e], mv));
        if (more) res[e] = __fadd_rn(res[e], __fmul_rn(next[e], mv));
    }
    if constexpr (N == 4) *reinterpret_cast<float4*>(out + at) = make_float4(res[0], res[1], res[2], res[3]);
    else out[at] = res[0];
}

// out [C, Rp] = FP16(+/-e)^T by the idx bits of stream-major words, rows R..Rp zero: the ROSA output (src/model.rs:1313) as
// the operand of a weight gradient.  A thread has eight rows of a column; blockIdx.y is the column.
__global__ void emit_transposed_kernel(const uint32_t* __restrict__ idx_sw, const uint16_t* __restrict__ e,
                                       uint16_t* __restrict__ out, uint32_t R, uint32_t C, uint32_t Rp, uint32_t time) {
    chain_entry();
    const uint32_t r0 = (blockIdx.x * blockDim.x + threadIdx.x) * 8u, c = blockIdx.y, wps = (time + 31u) / 32u;
    if (r0 >= Rp) return;
    uint32_t seq = r0 / time, t = r0 - seq * time, h[8];
    const uint32_t plus = e[c];
#pragma unroll
    for (uint32_t k = 0; k < 8u; ++k) {
        h[k] = 0u;
        if (r0 + k < R) h[k] = (idx_sw[((size_t)seq * C + c) * wps + (t >> 5)] >> (t & 31u)) & 1u ? plus : plus ^ 0x8000u;
        if (++t == time) { t = 0u; ++seq; }
    }
    *reinterpret_cast<uint4*>(out + (size_t)c * Rp + r0) =
        make_uint4(h[0] | h[1] << 16, h[2] | h[3] << 16, h[4] | h[5] << 16, h[6] | h[7] << 16);
}

// ------------------------------------------------------------ optimiser
// A CTA has 1024 elements, four per thread, their loads in flight together.  The gradient is the sum of `sums` arrays of n
// elements, in their order (the shares of a split product).
__global__ void __launch_bounds__(256)
clipped_sgd_kernel(uint16_t* __restrict__ w, float* __restrict__ residual, const float* __restrict__ g, uint32_t sums, float gmul,
                   float lr, size_t n) {
    chain_entry();
    const size_t i0 = (size_t)blockIdx.x * 1024 + threadIdx.x;
    uint16_t wb[4];
    float r[4], gv[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const size_t i = i0 + k * 256;
        if (i < n) { wb[k] = w[i]; r[k] = residual[i]; gv[k] = g[i]; }
    }
    for (uint32_t s = 1; s < sums; ++s) {
        g += n;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (i0 + k * 256 < n) gv[k] += g[i0 + k * 256];
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const size_t i = i0 + k * 256;
        if (i >= n) break;
        clipped_step(wb[k], r[k], __fmul_rn(gv[k], gmul), lr);
        w[i] = wb[k];
        residual[i] = r[k];
    }
}

// One latent (apply_binaryconnect_sgd, src/precision.rs:124-134); g not finite or zero: it stays.  True: something changed.
__device__ __forceinline__ bool latent_step(uint16_t& latent, float& residual, float g, float lr) {
    if (!(g != 0.0f && fabsf(g) <= 3.4028234e38f)) return false;
    const float update = __fmul_rn(lr, fminf(fmaxf(g, -1.0f), 1.0f));
    const float desired = fminf(fmaxf(__fadd_rn(__fsub_rn(h2f(latent), update), residual), -1.0f), 1.0f);
    latent = __half_as_ushort(__float2half_rn(desired));
    residual = __fsub_rn(desired, h2f(latent));
    return true;
}

// Latent step of a packed matrix (apply_binaryconnect_sgd, src/precision.rs:124-134, on
// g_w = scale[o] * G[o,i] * gmul * ste_scale), re-packing of the sign bits (rebinarize,
// src/model.rs:878-884) and the count of bits that changed.  A warp has LATENT_WORDS words of 32 elements, their loads
// in flight together; a CTA adds its count of changed bits once (an addition per word was up to 32 768 on one address:
// 38 us for a matrix of 1 M elements).
constexpr int LATENT_WORDS = 4;
__global__ void __launch_bounds__(256)
latent_sgd_kernel(uint16_t* __restrict__ latent, float* __restrict__ residual, const float* __restrict__ G,
                  const uint16_t* __restrict__ scale, uint32_t* __restrict__ bits, size_t out_f, size_t in_f,
                  float gmul, float ste_scale, float lr, unsigned long long* flips) {
    chain_entry();
    const int lane = threadIdx.x & 31;
    const size_t n = out_f * in_f, i0 = ((size_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * (32 * LATENT_WORDS) + lane;
    float g[LATENT_WORDS], carry[LATENT_WORDS];
    uint16_t lb[LATENT_WORDS];
    uint32_t old[LATENT_WORDS];
#pragma unroll
    for (int j = 0; j < LATENT_WORDS; ++j) {
        const size_t i = i0 + 32 * j;
        if (i < n) {
            const size_t o = n >> 32 ? i / in_f : (uint32_t)i / (uint32_t)in_f;
            g[j] = __fmul_rn(__fmul_rn(__fmul_rn(scale ? h2f(scale[o]) : 1.0f, G[i]), gmul), ste_scale);
            lb[j] = latent[i];
            carry[j] = residual[i];
            old[j] = bits ? bits[i >> 5] : 0u;
        }
    }
    uint32_t changed = 0;
#pragma unroll
    for (int j = 0; j < LATENT_WORDS; ++j) {
        const size_t i = i0 + 32 * j;
        bool plus = false;
        if (i < n) {
            if (latent_step(lb[j], carry[j], g[j], lr)) {
                residual[i] = carry[j];
                latent[i] = lb[j];
            }
            plus = h2f(lb[j]) >= 0.0f;
        }
        const uint32_t word = __ballot_sync(0xffffffffu, plus);
        if (bits && lane == 0 && i < n) {
            bits[i >> 5] = word;
            changed += __popc(old[j] ^ word);
        }
    }
    if (!flips) return;
    __shared__ uint32_t total;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    if (changed) atomicAdd(&total, changed);
    __syncthreads();
    if (threadIdx.x == 0 && total) atomicAdd(flips, (unsigned long long)total);
}

// All of a packed matrix's step after its gradient product: the sum of the product's shares (in their order), the latents
// as latent_sgd_kernel steps them (with the scale from before its own step), the signs, the count of those that changed, the
// gradient of the row's scale as g_scale_kernel sums it and the clipped step of that scale.  in_f is a multiple of 32.  A CTA
// has a row, each of its warps PACKED_WORDS words of it at a time; the first warp then adds up what they left, since the sum
// of a scale keeps its order (a lane's elements are 32 apart).  The loads of a share are in flight together.  On average
// over a step at 16 384 rows (512 x 512, 2048 x 512 and one 8192 x 512) as four kernels, G and the signs read twice and the
// sum of the shares written in between, 32 us, with a warp for a row 23, so 12.5.
constexpr int PACKED_WORDS = 4, PACKED_WARPS = 4;
__global__ void __launch_bounds__(32 * PACKED_WARPS)
packed_step_kernel(uint16_t* __restrict__ latent, float* __restrict__ residual, const float* __restrict__ G, uint32_t sums,
                   uint16_t* __restrict__ scale, float* __restrict__ scale_residual, uint32_t* __restrict__ bits, size_t n,
                   uint32_t in_f, float gmul, float ste_scale, float lr, unsigned long long* flips) {
    chain_entry();
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, o = blockIdx.x;
    __shared__ float terms[PACKED_WARPS * PACKED_WORDS][32];
    __shared__ uint32_t changed[PACKED_WARPS];
    uint16_t sw = scale[o];
    float sr = scale_residual[o], acc = 0.0f;
    const float s = h2f(sw);
    uint32_t flipped = 0;
    for (uint32_t i0 = 0; i0 < in_f; i0 += 32 * PACKED_WARPS * PACKED_WORDS) {
        const uint32_t here = min(PACKED_WARPS * PACKED_WORDS, (in_f - i0) >> 5);   // words of this round
        const size_t at = (size_t)o * in_f + i0 + warp * (32 * PACKED_WORDS) + lane;
        float g[PACKED_WORDS], carry[PACKED_WORDS];
        uint16_t lb[PACKED_WORDS];
        uint32_t old[PACKED_WORDS];
#pragma unroll
        for (int j = 0; j < PACKED_WORDS; ++j)
            if (warp * PACKED_WORDS + j < here) {
                g[j] = G[at + 32 * j];
                lb[j] = latent[at + 32 * j];
                carry[j] = residual[at + 32 * j];
                old[j] = bits[(at >> 5) + j];
            }
#pragma unroll 8
        for (uint32_t k = 1; k < sums; ++k) {
#pragma unroll
            for (int j = 0; j < PACKED_WORDS; ++j)
                if (warp * PACKED_WORDS + j < here) g[j] += G[k * n + at + 32 * j];
        }
#pragma unroll
        for (int j = 0; j < PACKED_WORDS; ++j) {
            if (warp * PACKED_WORDS + j >= here) break;
            terms[warp * PACKED_WORDS + j][lane] = (old[j] >> lane) & 1u ? g[j] : -g[j];
            if (latent_step(lb[j], carry[j], __fmul_rn(__fmul_rn(__fmul_rn(s, g[j]), gmul), ste_scale), lr)) {
                residual[at + 32 * j] = carry[j];
                latent[at + 32 * j] = lb[j];
            }
            const uint32_t word = __ballot_sync(0xffffffffu, h2f(lb[j]) >= 0.0f);
            if (lane == 0) bits[(at >> 5) + j] = word;
            flipped += __popc(old[j] ^ word);
        }
        __syncthreads();
        if (warp == 0)
            for (uint32_t j = 0; j < here; ++j) acc += terms[j][lane];
        __syncthreads();
    }
    if (lane == 0) changed[warp] = flipped;
    __syncthreads();
    if (warp) return;
    for (int k = 16; k > 0; k >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, k);
    if (lane == 0) {
        clipped_step(sw, sr, __fmul_rn(acc, gmul), lr);
        scale[o] = sw;
        scale_residual[o] = sr;
        uint32_t total = 0;
        for (int w = 0; w < PACKED_WARPS; ++w) total += changed[w];
        if (total) atomicAdd(flips, (unsigned long long)total);
    }
}

// g_scale[o] = sum_i sign[o,i] * G[o,i]   (g_scale of backward_ste, src/model.rs:784-790, with the
// row sum taken first).  One warp per output row.
__global__ void __launch_bounds__(256)
g_scale_kernel(const float* __restrict__ G, const uint32_t* __restrict__ bits, float* __restrict__ out, size_t out_f,
               size_t in_f) {
    chain_entry();
    const int lane = threadIdx.x & 31;
    const size_t o = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (o >= out_f) return;
    float acc = 0.0f;
    for (size_t i = lane; i < in_f; i += 32) {
        const size_t bit = o * in_f + i;
        const float g = G[bit];
        acc += (bits[bit >> 5] >> (bit & 31)) & 1u ? g : -g;
    }
    for (int k = 16; k > 0; k >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, k);
    if (lane == 0) out[o] = acc;
}

// Embedding rows: one clipped step per ROW in row order (src/model.rs:2980-2987), so a token that
// occurs n times is stepped n times.  A thread per (distinct token, channel).
// Bound by the chain of the most frequent token (a step is about 30 cycles, a tenth of what its gradient takes to arrive):
// the gradients of three batches of EMBED_BATCH occurrences are on their way to shared memory while one is worked on, and
// the rows they are in are read a batch earlier.  Each thread copies and reads its own channel alone.  16 384 Zipf(1.1)
// tokens of 8192, 512 channels: with the loads of eight occurrences at a time ahead of their steps 376 us, so 162.
constexpr int EMBED_BATCH = 16, EMBED_RING = 4, EMBED_THREADS = 128;
__global__ void __launch_bounds__(EMBED_THREADS)
embed_sgd_kernel(uint16_t* __restrict__ emb, float* __restrict__ residual, const float* __restrict__ gx,
                 const uint32_t* __restrict__ toks, const uint32_t* __restrict__ starts, const uint32_t* __restrict__ order,
                 size_t d, float gmul, float lr) {
    chain_entry();
    __shared__ float ring[EMBED_RING][EMBED_BATCH][EMBED_THREADS];
    const uint32_t tok = toks[blockIdx.x], r0 = starts[blockIdx.x], r1 = starts[blockIdx.x + 1];
    const size_t c = (size_t)blockIdx.y * EMBED_THREADS + threadIdx.x;
    if (c >= d) return;
    uint16_t wb = emb[(size_t)tok * d + c];
    float r = residual[(size_t)tok * d + c];
    uint32_t row[EMBED_BATCH] = {};   // of the batch that is fetched next
    // whole batches without a test per occurrence
    const auto rows_of = [&](uint32_t k0) {
        if (k0 + EMBED_BATCH <= r1) {
#pragma unroll
            for (int j = 0; j < EMBED_BATCH; ++j) row[j] = order[k0 + j];
        } else {
#pragma unroll
            for (int j = 0; j < EMBED_BATCH; ++j) if (k0 + j < r1) row[j] = order[k0 + j];
        }
    };
    const auto copy = [&](const float* slot, uint32_t from) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(slot)),
                     "l"(gx + (size_t)from * d + c) : "memory");
    };
    const auto fetch = [&](uint32_t k0) {
        float(*slot)[EMBED_THREADS] = ring[(k0 - r0) / EMBED_BATCH % EMBED_RING];
        if (k0 + EMBED_BATCH <= r1) {
#pragma unroll
            for (int j = 0; j < EMBED_BATCH; ++j) copy(&slot[j][threadIdx.x], row[j]);
        } else {
#pragma unroll
            for (int j = 0; j < EMBED_BATCH; ++j) if (k0 + j < r1) copy(&slot[j][threadIdx.x], row[j]);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll 1
    for (int k = 0; k < EMBED_RING - 1; ++k) {
        rows_of(r0 + k * EMBED_BATCH);
        fetch(r0 + k * EMBED_BATCH);
    }
    rows_of(r0 + (EMBED_RING - 1) * EMBED_BATCH);
#pragma unroll 1
    for (uint32_t k0 = r0; k0 < r1; k0 += EMBED_BATCH) {
        fetch(k0 + (EMBED_RING - 1) * EMBED_BATCH);   // an empty group past the end; its slot was read a batch ago
        rows_of(k0 + EMBED_RING * EMBED_BATCH);
        asm volatile("cp.async.wait_group %0;" ::"n"(EMBED_RING - 1) : "memory");
        const float(*slot)[EMBED_THREADS] = ring[(k0 - r0) / EMBED_BATCH % EMBED_RING];
        if (k0 + EMBED_BATCH <= r1) {
#pragma unroll
            for (int j = 0; j < EMBED_BATCH; ++j) clipped_step(wb, r, __fmul_rn(slot[j][threadIdx.x], gmul), lr);   // in row order
        } else {
            for (uint32_t j = 0; k0 + j < r1; ++j) clipped_step(wb, r, __fmul_rn(slot[j][threadIdx.x], gmul), lr);
        }
    }
    emb[(size_t)tok * d + c] = wb;
    residual[(size_t)tok * d + c] = r;
}

__global__ void init_latent_kernel(const uint32_t* __restrict__ bits, uint16_t* __restrict__ latent, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    latent[i] = (bits[i >> 5] >> (i & 31)) & 1u ? LATENT_PLUS : (uint16_t)(LATENT_PLUS | 0x8000u);
}

// The sums over chunks of rows, left in `part`.
void col_partial_launch(ullis_cuda_runtime* rt, const float* a, const void* b, float* part, size_t R, size_t C, ColMode mode, size_t time,
                        const float2* stats) {
    const size_t chunks = (R + COL_ROWS - 1) / COL_ROWS;
    const dim3 grid(blocks_for(C, 32), (unsigned)chunks);
    const auto run = [&](auto kernel) {
        rt->chain(kernel, grid, 256, 0, a, b, stats, part, (uint32_t)R, (uint32_t)C, (uint32_t)time);
    };
    switch (mode) {
        case COL_SUM: run(col_partial_kernel<COL_SUM>); break;
        case COL_LN: run(col_partial_kernel<COL_LN>); break;
        case COL_SHIFT: run(col_partial_kernel<COL_SHIFT>); break;
        case COL_SIGN: run(col_partial_kernel<COL_SIGN>); break;
        case COL_BITS: run(col_partial_kernel<COL_BITS>); break;
    }
    rt->launched("col_partial");
}
// out [outs, C], or the steps
void col_final_launch(ullis_cuda_runtime* rt, const float* part, float* out, size_t R, size_t C, unsigned outs, const ColStep& step) {
    rt->chain(col_final_kernel, dim3(blocks_for(C, 64), outs), 64, 0, part, out, (R + COL_ROWS - 1) / COL_ROWS, C, step);
    rt->launched("col_final");
}
// out [C] (COL_LN: two of them)
void col_reduce_launch(ullis_cuda_runtime* rt, const float* a, const void* b, float* out, size_t R, size_t C, ColMode mode,
                       DeviceBuffer& scratch, size_t time = 0, const float2* stats = nullptr) {
    const unsigned outs = mode == COL_LN ? 2 : 1;
    float* part = scratch.as<float>(outs * ((R + COL_ROWS - 1) / COL_ROWS) * C);
    col_partial_launch(rt, a, b, part, R, C, mode, time, stats);
    col_final_launch(rt, part, out, R, C, outs, ColStep{});
}

// ------------------------------------------------------------ host helpers
struct Step {
    ullis_cuda_train_state* st;
    ullis_cuda_runtime* rt;
    float gmul, lr, ste;

    // y [M,N] = a16 [M,K] . b16 [N,K]^T
    // (partials: or the shares that sum to it)
    void gemm(const uint16_t* a, const uint16_t* b, float* y, size_t M, size_t K, size_t N, tc::Partials* partials = nullptr) {
        if (tc::dense_nt(rt, a, b, y, M, K, N, partials)) return;
        if (partials) *partials = tc::Partials{y, 1};
        dim3 grid(blocks_for(N, 16), blocks_for(M, 16)), block(16, 16);
        gemm_nt_plain_kernel<<<grid, block, 0, rt->stream>>>(a, b, y, M, K, N);
        rt->launched("gemm_nt_plain");
    }
    // rows_out [R, pad64(C)] (or null) and t_out [C, Rp] of x [R, C]
    void operands(const float* x, const uint16_t* colscale, uint16_t* rows_out, uint16_t* t_out, size_t R, size_t C, size_t Rp) {
        const dim3 grid(blocks_for(Rp, 64), blocks_for(C, 64));
        rt->chain(operands_kernel<false>, grid, 256, 0, x, nullptr, colscale, rows_out, t_out, nullptr, R, C, pad64(C), Rp,
                  rt->dev_status);
        rt->launched("operands");
    }
    void operands_cmix(const float* g_relu2, const float* key, const uint16_t* colscale, uint16_t* rows_out, uint16_t* t_out,
                       uint16_t* relu2_t, size_t R, size_t C, size_t Rp) {
        const dim3 grid(blocks_for(Rp, 64), blocks_for(C, 64));
        rt->chain(operands_kernel<true>, grid, 256, 0, g_relu2, key, colscale, rows_out, t_out, relu2_t, R, C, pad64(C), Rp,
                  rt->dev_status);
        rt->launched("operands_cmix");
    }
    void unpack_transpose(const uint32_t* bits, uint16_t* out, size_t out_f, size_t in_f, size_t outp) {
        rt->chain(unpack_transpose_kernel, blocks_for(in_f * outp, 256), 256, 0, bits, out, out_f, in_f, outp);
        rt->launched("unpack_transpose");
    }
    // The gradient g[c] = sum_r f(a[r,c], b[r,c]) of a vector, and (after the last use of the vector, before the next gradient) its step.
    void col_gradient(const float* a, const void* b, size_t R, size_t C, ColMode mode, size_t time = 0, const float2* stats = nullptr) {
        col_partial_launch(rt, a, b, st->part.as<float>((mode == COL_LN ? 2 : 1) * ((R + COL_ROWS - 1) / COL_ROWS) * C), R, C, mode, time, stats);
    }
    void col_step(const Fp16Param& p, size_t R, float rate, const Fp16Param* second = nullptr) {
        col_final_launch(rt, st->part.as<float>(1), nullptr, R, p.n, second ? 2 : 1,
                         ColStep{{p.w, second ? second->w : nullptr}, {p.residual, second ? second->residual : nullptr}, gmul, rate});
    }
    void sgd(const Fp16Param& p, const float* g, float rate, uint32_t sums = 1) {
        rt->chain(clipped_sgd_kernel, blocks_for(p.n, 1024), 256, 0, p.w, p.residual, g, sums, gmul, rate, p.n);
        rt->launched("clipped_sgd");
    }
    // gx_out (+)= LN backward of (x, gy); steps the LayerNorm's weight and bias
    void ln_backward(const float* x, const float* gy, const Fp16Param& w, const Fp16Param& b, float* gx_out,
                     bool accumulate, size_t rows, size_t d) {
        float2* stats = st->ln_stats.as<float2>(rows);
        ln_backward_launch(rt, x, gy, w.w, gx_out, stats, rows, d, accumulate ? 1 : 0);
        col_gradient(gy, x, rows, d, COL_LN, 0, stats);   // g_weight, then g_bias
        col_step(w, rows, lr, &b);
    }
    // Packed matrix: G = gy^T . x (unscaled by the row scale), then scale / latent steps.
    // gy16t: FP16(gy)^T [out, rows_p]; x16t: FP16(x)^T [in, rows_p].
    void packed_update(PackedParam& p, const uint16_t* gy16t, const uint16_t* x16t, size_t rows_p, unsigned long long* flips, float* small) {
        const size_t out_f = p.weights->out, in_f = p.weights->in;
        float* G = st->gmat.as<float>(out_f * in_f);
        uint32_t* bits = const_cast<uint32_t*>(p.weights->bits);
        if (in_f % 32 == 0 && out_f < ((size_t)1 << 31)) {
            tc::Partials g{};
            gemm(gy16t, x16t, G, out_f, rows_p, in_f, &g);
            rt->chain(packed_step_kernel, (unsigned)out_f, 32 * PACKED_WARPS, 0, p.latent, p.latent_residual, g.sums, g.count,
                      p.scale.w, p.scale.residual, bits, out_f * in_f, (uint32_t)in_f, gmul, ste, lr, flips);
            rt->launched("packed_step");
        } else {   // a word has bits of two rows
            gemm(gy16t, x16t, G, out_f, rows_p, in_f);
            rt->chain(g_scale_kernel, blocks_for(out_f, 8), 256, 0, G, bits, small, out_f, in_f);
            rt->launched("g_scale");
            rt->chain(latent_sgd_kernel, blocks_for(out_f * in_f, 256 * LATENT_WORDS), 256, 0, p.latent, p.latent_residual, G,
                      p.scale.w, bits, out_f, in_f, gmul, ste, lr, flips);
            rt->launched("latent_sgd");
            sgd(p.scale, small, lr);
        }
    }
};

}  // namespace

// ------------------------------------------------------------ op-level launchers (kernels.hpp)
namespace ullis {
namespace k {

void clipped_sgd(ullis_cuda_runtime* rt, uint16_t* w, float* residual, const float* g, float lr, size_t n) {
    rt->chain(clipped_sgd_kernel, blocks_for(n, 1024), 256, 0, w, residual, g, 1u, 1.0f, lr, n);
    rt->launched("clipped_sgd");
}

void latent_sgd(ullis_cuda_runtime* rt, uint16_t* latent, float* residual, const float* g, float lr, float ste_scale,
                uint32_t* bits, size_t n) {
    rt->chain(latent_sgd_kernel, blocks_for(n, 256 * LATENT_WORDS), 256, 0, latent, residual, g, nullptr, bits, 1,
                                                                                  n, 1.0f, ste_scale, lr, nullptr);
    rt->launched("latent_sgd");
}

void rosa_e_grad(ullis_cuda_runtime* rt, const float* gy, const uint8_t* idx, float* g_e, size_t rows, size_t channels,
                 DeviceBuffer& scratch) {
    col_reduce_launch(rt, gy, idx, g_e, rows, channels, COL_SIGN, scratch);
}

void relu2_backward(ullis_cuda_runtime* rt, const float* input, float* g, size_t n) {
    rt->chain(relu2_bwd_kernel, blocks_for((n + 3) / 4, 256), 256, 0, input, g, n);
    rt->launched("relu2_bwd");
}

void layer_norm_backward(ullis_cuda_runtime* rt, const float* x, const float* gy, const uint16_t* w, float* gx,
                         float2* stats, float* gw_gb, size_t rows, size_t channels, DeviceBuffer& scratch) {
    ln_backward_launch(rt, x, gy, w, gx, stats, rows, channels, 0);
    col_reduce_launch(rt, gy, x, gw_gb, rows, channels, COL_LN, scratch, 0, stats);
}

}  // namespace k
}  // namespace ullis

// ------------------------------------------------------------ state
ullis_cuda_train_state::ullis_cuda_train_state(ullis_cuda_model* model, const uint8_t* checkpoint, size_t len)
    : m(model), rt(model->rt) {
    rt->bind();
    const size_t d = m->d, f = m->ffn, v = m->vocab;
    layers.assign(m->layers, Layer{});
    // plan: every latent (u16) and residual (f32) in one zeroed allocation
    struct Slot { void** at; size_t bytes; size_t offset; };
    std::vector<Slot> slots;
    size_t total = 0;
    auto want = [&](void** at, size_t bytes) {
        slots.push_back({at, bytes, total});
        total = (total + bytes + 255) / 256 * 256;
    };
    auto fp16 = [&](Fp16Param& p, const uint16_t* w, size_t n, const std::string& name) {
        p.w = const_cast<uint16_t*>(w);
        p.n = n;
        want(reinterpret_cast<void**>(&p.residual), n * 4);
        named[name] = Named{p.w, n * 2};
    };
    auto packed = [&](PackedParam& p, PackedWeights& w, const std::string& name) {
        p.weights = &w;
        const size_t n = w.out * w.in;
        want(reinterpret_cast<void**>(&p.latent), n * 2);
        want(reinterpret_cast<void**>(&p.latent_residual), n * 4);
        fp16(p.scale, w.scale, w.out, name + ".scale");
        if (w.bias) fp16(p.bias, w.bias, w.out, name + ".bias");
        named[name + ".bits"] = Named{const_cast<uint32_t*>(w.bits), (n + 31) / 32 * 4};
    };
    fp16(embedding, m->embedding, v * d, "embedding");
    fp16(ln_out_w, m->ln_out.weight, d, "ln_out.weight");
    fp16(ln_out_b, m->ln_out.bias, d, "ln_out.bias");
    packed(head, m->head, "head");
    for (size_t l = 0; l < m->layers; ++l) {
        LayerWeights& L = m->blocks[l];
        Layer& T = layers[l];
        const std::string pre = "blocks." + std::to_string(l);
        if (l == 0) {
            fp16(T.ln0_w, L.ln0.weight, d, pre + ".ln0.weight");
            fp16(T.ln0_b, L.ln0.bias, d, pre + ".ln0.bias");
        }
        fp16(T.ln2_w, L.ln2.weight, d, pre + ".ln2.weight");
        fp16(T.ln2_b, L.ln2.bias, d, pre + ".ln2.bias");
        fp16(T.e, L.e, d, pre + ".rosa.e");
        fp16(T.x_k, L.ffn_x_k, d, pre + ".ffn.x_k");
        fp16(T.value, L.value, f * d, pre + ".ffn.value");
        packed(T.o, L.o, pre + ".rosa.o");
        packed(T.key, L.key, pre + ".ffn.key");
        // frozen in this mode, readable all the same
        named[pre + ".rosa.q.bits"] = Named{const_cast<uint32_t*>(L.q.bits), (d * d + 31) / 32 * 4};
        named[pre + ".rosa.k.bits"] = Named{const_cast<uint32_t*>(L.k.bits), (d * d + 31) / 32 * 4};
        named[pre + ".rosa.v.bits"] = Named{const_cast<uint32_t*>(L.v.bits), (d * d + 31) / 32 * 4};
        named[pre + ".ln3.weight"] = Named{const_cast<uint16_t*>(L.ln3.weight), d * 2};
        named[pre + ".rosa.x_q"] = Named{const_cast<uint16_t*>(L.x_q), d * 2};
    }
    uint8_t* base = static_cast<uint8_t*>(carry.ensure(total ? total : 256));
    rt->zero(base, total);
    for (const Slot& s : slots) *s.at = base + s.offset;

    // latents: +/-0.01 by the sign bit (src/model.rs:640-649) unless the checkpoint carries them
    auto init_latent = [&](PackedParam& p, const std::string& name) {
        const size_t n = p.weights->out * p.weights->in;
        init_latent_kernel<<<blocks_for(n, 256), 256, 0, rt->stream>>>(p.weights->bits, p.latent, n);
        rt->launched("init_latent");
        named[name + ".latent"] = Named{p.latent, n * 2};
        named[name + ".latent.residual"] = Named{p.latent_residual, n * 4};
    };
    init_latent(head, "head");
    for (size_t l = 0; l < m->layers; ++l) {
        init_latent(layers[l].o, "blocks." + std::to_string(l) + ".rosa.o");
        init_latent(layers[l].key, "blocks." + std::to_string(l) + ".ffn.key");
    }
    auto residual_name = [&](const Fp16Param& p, const std::string& name) {
        named[name + ".residual"] = Named{p.residual, p.n * 4};
    };
    residual_name(embedding, "embedding");
    residual_name(ln_out_w, "ln_out.weight");
    residual_name(ln_out_b, "ln_out.bias");
    residual_name(head.scale, "head.scale");
    if (head.bias.w) residual_name(head.bias, "head.bias");
    for (size_t l = 0; l < m->layers; ++l) {
        Layer& T = layers[l];
        const std::string pre = "blocks." + std::to_string(l);
        if (l == 0) {
            residual_name(T.ln0_w, pre + ".ln0.weight");
            residual_name(T.ln0_b, pre + ".ln0.bias");
        }
        residual_name(T.ln2_w, pre + ".ln2.weight");
        residual_name(T.ln2_b, pre + ".ln2.bias");
        residual_name(T.e, pre + ".rosa.e");
        residual_name(T.x_k, pre + ".ffn.x_k");
        residual_name(T.value, pre + ".ffn.value");
        residual_name(T.o.scale, pre + ".rosa.o.scale");
        if (T.o.bias.w) residual_name(T.o.bias, pre + ".rosa.o.bias");
        residual_name(T.key.scale, pre + ".ffn.key.scale");
    }
    // carry of a resumed run: "<name>.latent" (F16) and "<name>.residual" (F32) tensors
    // (src/model.rs:3461-3466, 3724-3740)
    if (checkpoint && len) {
        SafeTensors stf = parse_safetensors(checkpoint, len);
        for (const auto& kv : stf.tensors) {
            const std::string& name = kv.first;
            const bool is_latent = name.size() > 7 && name.compare(name.size() - 7, 7, ".latent") == 0;
            const bool is_residual = name.size() > 9 && name.compare(name.size() - 9, 9, ".residual") == 0;
            if (!is_latent && !is_residual) continue;
            auto it = named.find(name);
            if (it == named.end()) continue;   // carry of a tensor this mode does not step
            if (kv.second.dtype != (is_latent ? "F16" : "F32") || kv.second.bytes != it->second.bytes)
                fail(ULLIS_CUDA_ERR_CHECKPOINT, "checkpoint carry shape mismatch (" + name + ")");
            rt->h2d(it->second.ptr, kv.second.data, kv.second.bytes);
        }
    }
    rt->sync();
}

void ullis_cuda_train_state::read(const char* name, void* dst, size_t bytes) {
    auto it = named.find(name ? name : "");
    if (it == named.end()) fail(ULLIS_CUDA_ERR_ARG, std::string("unknown tensor ") + (name ? name : "(null)"));
    if (bytes != it->second.bytes)
        fail(ULLIS_CUDA_ERR_SHAPE, "tensor size mismatch: expected " + std::to_string(it->second.bytes) + " bytes");
    rt->bind();
    rt->d2h(dst, it->second.ptr, bytes);
    rt->sync();
}

// ------------------------------------------------------------ the step
void ullis_cuda_train_state::step(const uint32_t* tokens, const uint32_t* labels_h, uint32_t ignore_id, size_t batch,
                                  size_t time, float learning_rate, ullis_cuda_train_result* out) {
    // src/model.rs:2837-2861
    if (!std::isfinite(learning_rate) || learning_rate <= 0.0f || time < 2)
        fail(ULLIS_CUDA_ERR_ARG, "train step requires a positive learning rate and time >= 2");
    if (!tokens || !labels_h) fail(ULLIS_CUDA_ERR_ARG, "tokens or labels is null");
    m->check_shape(batch, time);
    const size_t d = m->d, f = m->ffn, vocab = m->vocab, rows = batch * time;
    for (size_t r = 0; r < rows; ++r)
        if (tokens[r] >= vocab || (labels_h[r] != ignore_id && labels_h[r] >= vocab))
            fail(ULLIS_CUDA_ERR_SHAPE, "token shape or context length is invalid");
    rt->bind();

    // rows of each distinct token, in row order, for the embedding step
    std::vector<uint32_t> count(vocab + 1, 0), h_order(rows), h_toks, h_starts;
    for (size_t r = 0; r < rows; ++r) ++count[tokens[r] + 1];
    for (size_t t = 0; t < vocab; ++t) count[t + 1] += count[t];
    {
        std::vector<uint32_t> at(count.begin(), count.end() - 1);
        for (size_t r = 0; r < rows; ++r) h_order[at[tokens[r]]++] = (uint32_t)r;
    }
    for (size_t t = 0; t < vocab; ++t)
        if (count[t + 1] != count[t]) {
            h_toks.push_back((uint32_t)t);
            h_starts.push_back(count[t]);
        }
    h_starts.push_back((uint32_t)rows);
    rt->h2d(order.as<uint32_t>(rows), h_order.data(), rows * 4);
    rt->h2d(toks.as<uint32_t>(h_toks.size()), h_toks.data(), h_toks.size() * 4);
    rt->h2d(starts.as<uint32_t>(h_starts.size()), h_starts.data(), h_starts.size() * 4);

    // forward with the tape
    m->upload_tokens(tokens, labels_h, batch, time);
    m->train_tape = true;
    try {
        m->enqueue_hidden(batch, time);
    } catch (...) {
        m->train_tape = false;
        throw;
    }
    m->train_tape = false;

    const size_t n = rows * d, rows_p = pad64(rows), vocab_p = pad64(vocab), d_p = pad64(d), f_p = pad64(f);
    const bool exact = rt->mode == ULLIS_CUDA_MODE_EXACT;
    float P = 1.0f;
    while (P < (float)(time - 1)) P *= 2.0f;
    Step s{this, rt, 1.0f / P, learning_rate, (float)(time - 1)};
    float* X = m->x.as<float>(n);        // residual stream before ln_out
    float* H = m->a.as<float>(n);        // ln_out(X)
    float* GX = gx.as<float>(n);
    float* T1 = t1.as<float>(n);
    float* T2 = t2.as<float>(n);
    float* T3 = t3.as<float>(n);
    float* W1 = wide1.as<float>(rows * f);
    float* W2 = wide2.as<float>(rows * f);
    float* LG = logits.as<float>(rows * vocab);
    const size_t widest = std::max({f_p, vocab_p, d_p});
    uint16_t* A16 = a16.as<uint16_t>(rows * widest);
    uint16_t* B16 = b16.as<uint16_t>(std::max(d * rows_p, widest * std::max(f, d)));
    uint16_t* T16 = t16.as<uint16_t>(std::max(vocab, d + 2 * f) * rows_p);
    float* SM = small.as<float>(std::max({f, vocab, d}));   // gradients of a packed matrix's scales
    unsigned long long* CNT = counters.as<unsigned long long>(3);
    const uint32_t* lab = m->labels.as<uint32_t>(rows);
    float* RL = m->row_loss.as<float>(rows);
    uint8_t* res = static_cast<uint8_t*>(m->result.ensure(16));
    rt->zero(CNT, 24);
    gmat.as<float>(std::max({d * f, vocab * d, d * d}));                        // sized once: no growth mid-step
    part.as<float>((rows + 255) / 256 * std::max({f, vocab, 2 * d}));

    // ---- head: logits, loss, gy (src/model.rs:3204-3257)
    if (!tc::binary_linear(rt, H, m->head.bits, m->head.scale, m->head.bias, LG, rows, d, vocab))
        k::binary_linear_exact(rt, H, m->head.bits, m->head.scale, m->head.bias, LG, rows, d, vocab, false);
    rt->chain(ce_grad_kernel, (unsigned)rows, 256, 0, LG, lab, ignore_id, rows, time, vocab,
                                                          1.0f / (float)(time - 1), P, RL, rt->dev_status);
    rt->launched("ce_grad");
    k::ce_reduce(rt, RL, lab, ignore_id, rows, time, reinterpret_cast<double*>(res),
                 reinterpret_cast<unsigned long long*>(res + 8));
    m->have_result = true;
    if (head.bias.w) {   // not used again in this step
        s.col_gradient(LG, nullptr, rows, vocab, COL_SUM);
        s.col_step(head.bias, rows, learning_rate * HEAD_BIAS_LR_MULT);
    }
    s.operands(LG, m->head.scale, A16, T16, rows, vocab, rows_p);                   // (gy*scale) [rows, V], gy^T [V, rows]
    s.unpack_transpose(m->head.bits, B16, vocab, d, vocab_p);                       // S^T [d, V]
    s.gemm(A16, B16, GX, rows, vocab_p, d);                                         // g_hidden
    s.operands(H, nullptr, nullptr, B16, rows, d, rows_p);                          // hidden^T [d, rows]
    s.packed_update(head, T16, B16, rows_p, CNT + 0, SM);

    // ---- ln_out
    s.ln_backward(X, GX, ln_out_w, ln_out_b, T1, false, rows, d);
    std::swap(GX, T1);

    for (size_t li = m->layers; li-- > 0;) {
        LayerWeights& L = m->blocks[li];
        Layer& T = layers[li];
        const float* AR = m->tape_after[li].as<float>(n);   // residual stream after the ROSA block
        // ---- CMix: recompute ln2 -> shifted -> key from the tape (src/model.rs:1050-1061)
        k::layer_norm(rt, AR, L.ln2.weight, L.ln2.bias, T1, rows, d, exact);
        k::shift_mix(rt, T1, L.ffn_x_k, nullptr, nullptr, T2, nullptr, nullptr, rows, time, d);     // shifted
        if (!tc::binary_linear(rt, T2, L.key.bits, L.key.scale, nullptr, W1, rows, d, f))
            k::binary_linear_exact(rt, T2, L.key.bits, L.key.scale, nullptr, W1, rows, d, f, false);  // key
        // value: g_relu2 = gy . W (before W is stepped), g_W = gy^T . relu2 (src/model.rs:1138-1140)
        uint16_t *key_t = T16 + d * rows_p, *relu2_t = key_t + f * rows_p;
        s.operands(GX, nullptr, A16, T16, rows, d, rows_p);                                           // gy, gy^T
        rt->chain(transpose16_kernel, dim3(blocks_for(d_p, 64), blocks_for(f, 64)), 256, 0, L.value, B16, d, f, d_p);
        rt->launched("transpose16");
        // g_relu2 and what the products of the key take of it: in one kernel where that goes, which reads A16 while it writes
        uint16_t* KEY16 = reinterpret_cast<uint16_t*>(W2);
        if (!tc::cmix_grad_operands(rt, A16, B16, W1, L.key.scale, KEY16, key_t, relu2_t, rows, d_p, f, rows_p)) {
            KEY16 = A16;
            s.gemm(A16, B16, W2, rows, d_p, f);
            s.operands_cmix(W2, W1, L.key.scale, KEY16, key_t, relu2_t, rows, f, rows_p);
        }
        {
            float* G = gmat.as<float>(d * f);
            tc::Partials g{};
            s.gemm(T16, relu2_t, G, d, rows_p, f, &g);
            s.sgd(T.value, g.sums, learning_rate, g.count);
        }
        // key (src/model.rs:1141-1163)
        s.unpack_transpose(L.key.bits, B16, f, d, f_p);
        s.gemm(KEY16, B16, T3, rows, f_p, d);                                                         // g_shifted
        s.operands(T2, nullptr, nullptr, B16, rows, d, rows_p);
        s.packed_update(T.key, key_t, B16, rows_p, CNT + 1, SM);
        // time-shift mix (src/model.rs:1164-1176)
        s.col_gradient(T3, T1, rows, d, COL_SHIFT, time);                                                       // g_mix
        if (d % 4 == 0)
            rt->chain(lerp_bwd_kernel<4>, blocks_for(n / 4, 256), 256, 0, T3, L.ffn_x_k, T1, (uint32_t)rows, (uint32_t)time,
                      (uint32_t)d);
        else
            rt->chain(lerp_bwd_kernel<1>, blocks_for(n, 256), 256, 0, T3, L.ffn_x_k, T1, (uint32_t)rows, (uint32_t)time, (uint32_t)d);
        rt->launched("lerp_bwd");
        s.col_step(T.x_k, rows, learning_rate);                                                       // after its last use
        s.ln_backward(AR, T1, T.ln2_w, T.ln2_b, GX, true, rows, d);

        // ---- ROSA: gradients stop at the q/k/v bits (src/model.rs:1494-1521)
        const uint32_t* idx = m->tape_idx[li].as<uint32_t>(1);
        if (T.o.bias.w) {   // not used again in this step
            s.col_gradient(GX, nullptr, rows, d, COL_SUM);
            s.col_step(T.o.bias, rows, learning_rate);
        }
        s.operands(GX, L.o.scale, A16, T16, rows, d, rows_p);
        s.unpack_transpose(L.o.bits, B16, d, d, d_p);
        s.gemm(A16, B16, T2, rows, d_p, d);                                                           // g_y
        s.col_gradient(T2, idx, rows, d, COL_BITS, time);                                             // g_e
        rt->chain(emit_transposed_kernel, dim3(blocks_for(rows_p, 8 * 128), (unsigned)d), 128, 0, idx, L.e, B16, (uint32_t)rows,
                  (uint32_t)d, (uint32_t)rows_p, (uint32_t)time);                                      // y = +/-e
        rt->launched("emit_transposed");
        s.col_step(T.e, rows, learning_rate);                                                         // after its last use
        s.packed_update(T.o, T16, B16, rows_p, CNT + 2, SM);

        if (li == 0) {   // ln0 replaced x on layer 0: its input is the embedded rows (src/model.rs:2972-2977)
            k::embed(rt, m->ids.as<uint32_t>(rows), m->embedding, T1, rows, d, vocab);
            s.ln_backward(T1, GX, T.ln0_w, T.ln0_b, T2, false, rows, d);
            std::swap(GX, T2);
        }
    }
    // ---- embedding rows (src/model.rs:2980-2987)
    rt->chain(embed_sgd_kernel, dim3((unsigned)h_toks.size(), blocks_for(d, EMBED_THREADS)), EMBED_THREADS, 0, embedding.w, embedding.residual, GX,
                                                                      toks.as<uint32_t>(1), starts.as<uint32_t>(1),
                                                                      order.as<uint32_t>(1), d, s.gmul, learning_rate);
    rt->launched("embed_sgd");

    unsigned long long h_cnt[3] = {0, 0, 0};
    rt->d2h(h_cnt, CNT, 24);
    float mean = 0.0f;
    uint64_t n_valid = 0;
    m->read_loss(&mean, nullptr, &n_valid, nullptr, 0);   // synchronises and checks the status word
    ++steps;
    if (out) *out = ullis_cuda_train_result{mean, n_valid, h_cnt[0], h_cnt[1], h_cnt[2]};
}

// install_head_unigram_prior (src/model.rs:3034-3085) with shrink_head_kaiming_scale (3087-3110): a
// one-shot host computation over the labels and two vocabulary-sized tensors.
void ullis_cuda_train_state::install_head_unigram_prior(const uint32_t* labels, size_t n, uint32_t ignore_id,
                                                        ullis_cuda_head_unigram_install* out) {
    if (!labels && n) fail(ULLIS_CUDA_ERR_ARG, "labels is null");
    const size_t vocab = m->vocab, d = m->d;
    rt->bind();
    std::vector<uint16_t> bias(vocab), scale(vocab);
    rt->d2h(bias.data(), head.bias.w, vocab * 2);
    rt->d2h(scale.data(), head.scale.w, vocab * 2);
    rt->sync();
    auto to_f32 = [](uint16_t b) { return __half2float(__ushort_as_half(b)); };
    auto to_f16 = [](float v) { return __half_as_ushort(__float2half_rn(v)); };
    auto rms = [&](const std::vector<uint16_t>& v) {
        float sum_sq = 0.0f;
        for (uint16_t b : v) sum_sq += to_f32(b) * to_f32(b);
        return v.empty() ? 0.0f : std::sqrt(sum_sq / (float)v.size());
    };
    float abs_sum = 0.0f;
    for (uint16_t b : bias) abs_sum += std::fabs(to_f32(b));
    ullis_cuda_head_unigram_install r{};
    if (abs_sum / (float)vocab > 0.05f) {   // HEAD_BIAS_PRIOR_ABS_EPS: a fitted prior is left alone
        r.bias_rms = rms(bias);
        r.scale_rms = rms(scale);
        if (out) *out = r;
        return;
    }
    std::vector<uint64_t> counts(vocab, 0);
    uint64_t n_targets = 0;
    for (size_t i = 0; i < n; ++i) {
        if (labels[i] == ignore_id || labels[i] >= vocab) continue;
        ++counts[labels[i]];
        ++n_targets;
    }
    if (n_targets == 0) fail(ULLIS_CUDA_ERR_ARG, "head unigram prior needs at least one supervised label");
    const float log_denom = std::log((float)n_targets + (float)vocab);
    std::vector<float> logs(vocab);
    float log_sum = 0.0f;
    for (size_t v = 0; v < vocab; ++v) {
        logs[v] = std::log1p((float)counts[v]) - log_denom;
        log_sum += logs[v];
    }
    const float log_mean = log_sum / (float)vocab;
    for (size_t v = 0; v < vocab; ++v) bias[v] = to_f16(logs[v] - log_mean);
    std::vector<float> zeros(vocab, 0.0f);
    rt->h2d(head.bias.w, bias.data(), vocab * 2);
    rt->h2d(head.bias.residual, zeros.data(), vocab * 4);   // Fp16Storage::set clears the carry (src/precision.rs:208-211)
    const float kaiming = 1.0f / std::sqrt((float)d);
    float mean = 0.0f;
    for (uint16_t b : scale) mean += to_f32(b);
    mean /= (float)vocab;
    if (mean > kaiming * 0.5f && mean < kaiming * 2.0f) {
        for (uint16_t& b : scale) b = to_f16(to_f32(b) * 0.25f);   // HEAD_KAIMING_SCALE_SHRINK
        rt->h2d(head.scale.w, scale.data(), vocab * 2);
        rt->h2d(head.scale.residual, zeros.data(), vocab * 4);
        r.shrunk_kaiming_scale = 1;
    }
    rt->sync();
    r.applied = 1;
    r.n_targets = n_targets;
    r.bias_rms = rms(bias);
    r.scale_rms = rms(scale);
    if (out) *out = r;
}
