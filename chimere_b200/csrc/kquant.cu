// Plain GEMV on K-quant super-blocks (Q4_K, Q5_K, Q6_K) against one Q8_1 row: the entries chimere_mmvq_q4k / _q5k / _q6k
// that the reference binds to its dependency's mul_mat_vec_*_K_q8_1 kernels (ffi/ggml_cuda_gemv.cu:118-172).  The
// production files keep the shared expert in Q5_K (moe_ffn.rs:1597-1650); the routed experts never use these types.
//
// A warp owns one output row (and up to eight input rows).  Lane l takes the 32-weight sub-blocks l, l+32, ... of the row:
// it reads the sub-block's quants as eight 32-bit words once, the Q8_1 block of every input row beside it, and adds
//     d * d8 * sc_j * dot - dmin * m_j * s8        (Q4_K, Q5_K: six-bit scale sc_j and min m_j, s8 = d8 * sum of the quants)
//     d * d8 * (sc_a * dot_a + sc_b * dot_b)       (Q6_K: one int8 scale per 16 weights)
// in ascending sub-block order; the lanes' sums meet in a butterfly.  HBM-bound: a row is read once, coalesced by
// super-block (consecutive lanes read consecutive 32-weight pieces), the Q8_1 row stays in L1/L2.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "common.cuh"
#include "kernels.h"
#include "kquant.cuh"

namespace chimere {

namespace {

constexpr int kRowsPerCta = 8;   // warps per CTA

// grid = (row groups, groups of tpc <= kTokensPerCta input rows, matrices).  A sub-block is decoded once and used for every input
// row of the CTA's group.  mode 0: y = v; 1: y += v; 2: y += sigmoid(logit[t]) * v (the sigmoid-gated shared expert added
// to the routed sum, scratch_pool.rs:266-277).  blockIdx.z = 1 takes the second matrix / output (gate beside up).
constexpr int kTokensPerCta = 8;
template <int TYPE>
__global__ void __launch_bounds__(32 * kRowsPerCta) kquant_mmvq_kernel(const uint8_t* w, const uint8_t* w2, const uint8_t* xq8, int64_t x_stride, float* y,
                                                                      float* y2, int64_t y_stride, int n_inputs, int tpc, int ncols, int nrows, int mode,
                                                                      const float* logit) {
    const int lane = threadIdx.x & 31, row = blockIdx.x * kRowsPerCta + (threadIdx.x >> 5);
    const int t0 = blockIdx.y * tpc, nt = min(tpc, n_inputs - t0);   // tpc <= kTokensPerCta input rows per CTA
    griddep_wait();   // (a no-op unless launched programmatically behind the kernel that writes the inputs)
    if (threadIdx.x == 0) griddep_launch();
    if (row >= nrows) return;
    if (blockIdx.z) { w = w2; y = y2; }
    const int nsub = ncols >> 5;
    const uint8_t* rowp = w + (size_t)row * (size_t)(ncols >> 8) * KBlock<TYPE>::kBytes;
    const uint8_t* xr = xq8 + (size_t)t0 * x_stride;
    float acc[kTokensPerCta];
#pragma unroll
    for (int i = 0; i < kTokensPerCta; ++i) acc[i] = 0.0f;
    for (int sb = lane; sb < nsub; sb += 32) {
        SubBlock s;
        decode_sub<TYPE>(rowp + (size_t)(sb >> 3) * KBlock<TYPE>::kBytes, sb & 7, s);
#pragma unroll
        for (int i = 0; i < kTokensPerCta; ++i)
            if (i < nt) acc[i] = add_dot<TYPE>(acc[i], s, xr + (size_t)i * x_stride + (size_t)sb * kQ81Bytes);
    }
#pragma unroll
    for (int i = 0; i < kTokensPerCta; ++i) {
        if (i < nt) {
            float v = acc[i];
#pragma unroll
            for (int sft = 16; sft > 0; sft >>= 1) v += __shfl_xor_sync(0xffffffffu, v, sft);
            if (lane == 0) {
                float* out = y + (size_t)(t0 + i) * y_stride + row;
                if (mode == 0) *out = v;
                else if (mode == 1) *out = v + *out;
                else *out = fmaf(v, sigmoid_ref(logit[t0 + i]), *out);
            }
        }
    }
}

// One warp per (row t, block b of 32): v = silu(g) * u (or relu(u)^2 without a gate row) -> one Q8_1 block, as the gate/up
// kernels write their intermediates (d = amax / 127 in f16, s = the sum of the 32 values).
__global__ void __launch_bounds__(256) act_q8_1_kernel(const float* g, const float* u, int64_t in_stride, uint8_t* out, int64_t out_stride, int T, int F) {
    const int lane = threadIdx.x & 31, nb = F >> 5;
    const int64_t wid = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    griddep_wait();
    if (threadIdx.x == 0) griddep_launch();
    if (wid >= (int64_t)T * nb) return;
    const int t = (int)(wid / nb), b = (int)(wid - (int64_t)t * nb);
    const float uu = u[(size_t)t * in_stride + b * 32 + lane];
    float v;
    if (g) v = silu_mul_ref(g[(size_t)t * in_stride + b * 32 + lane], uu);
    else { const float r = fmaxf(uu, 0.0f); v = r * r; }
    float amax = fabsf(v), sum = v;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, s));
        sum += __shfl_xor_sync(0xffffffffu, sum, s);
    }
    const float d = amax / 127.0f;
    uint8_t* blk = out + (size_t)t * out_stride + (size_t)b * kQ81Bytes;
    reinterpret_cast<int8_t*>(blk)[4 + lane] = (amax == 0.0f) ? (int8_t)0 : (int8_t)roundf(v / d);
    if (lane == 0) *reinterpret_cast<__half2*>(blk) = __halves2half2(__float2half(d), __float2half(sum));
}

// Q4_K / Q5_K rows -> the grouped GEMM's operand with minimums: per (128-row tile, stage of four 32-weight sub-blocks) four mma128
// tiles (int8 quants, words of f16 d << 16 | sc) and then [4][128] f32 -dmin * m * 2^-49 (the power of two the GEMM's sums carry).  mode as for
// the plain operand: 0 rows as they are, 1 / 2 gate / up rows interleaved per 64 and sub-blocks in tree order (operand_min_block).
// One thread per (row, sub-block).
template <int TYPE>
__global__ void __launch_bounds__(256) pack_operand_min_kernel(const uint8_t* __restrict__ raw, uint8_t* __restrict__ out, int nrows, int ncols, int mode) {
    const int nb = ncols >> 5;
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)nrows * nb) return;
    const int r = (int)(idx % nrows), b = (int)(idx / nrows);
    SubBlock s;
    decode_sub<TYPE>(raw + ((size_t)r * (ncols >> 8) + (b >> 3)) * KBlock<TYPE>::kBytes, b & 7, s);
    const int dr = mode == 0 ? r : (r >> 6) * 128 + (r & 63) + (mode == 2 ? 64 : 0);
    const int at = mode == 0 ? b : operand_min_block(b, nb), tile = dr >> 7, rr = dr & 127, u = at & 3;
    uint8_t* stage = out + ((size_t)tile * (nb >> 2) + (at >> 2)) * kOperandMinStage;
    uint8_t* dst = stage + u * 4608;
    *reinterpret_cast<uint4*>(dst + (rr >> 3) * 128 + (rr & 7) * 16) = make_uint4(s.w[0], s.w[1], s.w[2], s.w[3]);
    *reinterpret_cast<uint4*>(dst + 2048 + (rr >> 3) * 128 + (rr & 7) * 16) = make_uint4(s.w[4], s.w[5], s.w[6], s.w[7]);
    *reinterpret_cast<uint32_t*>(dst + 4096 + rr * 4) = ((uint32_t)__half_as_ushort(__float2half(s.d)) << 16) | (uint32_t)s.sc;
    *reinterpret_cast<float*>(stage + 4 * 4608 + u * 512 + rr * 4) = -(s.dmin * (float)s.mn) * __uint_as_float(0x27000000u);   // 2^-49
}

}  // namespace

cudaError_t launch_pack_operand_min(int type, const void* raw, void* out, int nrows, int ncols, int mode, cudaStream_t stream) {
    const int64_t n = (int64_t)nrows * (ncols / 32);
    if (n <= 0 || ncols % 256) return cudaErrorInvalidValue;
    const unsigned grid = (unsigned)((n + 255) / 256);
    if (type == CHIMERE_TYPE_Q4_K) pack_operand_min_kernel<CHIMERE_TYPE_Q4_K><<<grid, 256, 0, stream>>>((const uint8_t*)raw, (uint8_t*)out, nrows, ncols, mode);
    else if (type == CHIMERE_TYPE_Q5_K) pack_operand_min_kernel<CHIMERE_TYPE_Q5_K><<<grid, 256, 0, stream>>>((const uint8_t*)raw, (uint8_t*)out, nrows, ncols, mode);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

// w2 / y2 (optional): a second matrix of the same type and shape against the same inputs, in the same launch.
// chained: launch programmatically behind the previous kernel of the stream.
cudaError_t launch_mmvq_kquant_batched(int wtype, const void* w, const void* w2, const void* xq8, int64_t x_stride, float* y, float* y2,
                                       int64_t y_stride, int n_inputs, int ncols, int nrows, int mode, const float* logit, bool chained,
                                       cudaStream_t stream) {
    if (nrows <= 0 || n_inputs <= 0) return cudaSuccess;
    if (ncols <= 0 || (ncols & 255) || ((uintptr_t)xq8 & 3) || (x_stride & 3) || n_inputs > 65535 || (mode == 2 && !logit)) return cudaErrorInvalidValue;
    const uintptr_t wbits = (uintptr_t)w | (uintptr_t)w2;
    // input rows per CTA: as many as still leave a grid of two CTAs per SM (a small batch wants the CTAs, a large one the reuse)
    const int row_groups = (nrows + kRowsPerCta - 1) / kRowsPerCta;
    int tpc = kTokensPerCta;
    while (tpc > 1 && (int64_t)row_groups * ((n_inputs + tpc - 1) / tpc) * (w2 ? 2 : 1) < 2 * sm_count()) tpc >>= 1;
    const dim3 grid(row_groups, (n_inputs + tpc - 1) / tpc, w2 ? 2 : 1);
    const uint8_t* wp = (const uint8_t*)w;
    const uint8_t* wp2 = (const uint8_t*)w2;
    const uint8_t* xp = (const uint8_t*)xq8;
    auto go = [&](auto kernel) {
        if (chained) return launch_pdl(kernel, grid, 32 * kRowsPerCta, 0, stream, wp, wp2, xp, x_stride, y, y2, y_stride, n_inputs, tpc, ncols, nrows, mode, logit);
        kernel<<<grid, 32 * kRowsPerCta, 0, stream>>>(wp, wp2, xp, x_stride, y, y2, y_stride, n_inputs, tpc, ncols, nrows, mode, logit);
        return cudaGetLastError();
    };
    switch (wtype) {
        case CHIMERE_TYPE_Q4_K: return (wbits & 3) ? cudaErrorInvalidValue : go(kquant_mmvq_kernel<CHIMERE_TYPE_Q4_K>);
        case CHIMERE_TYPE_Q5_K: return (wbits & 3) ? cudaErrorInvalidValue : go(kquant_mmvq_kernel<CHIMERE_TYPE_Q5_K>);
        case CHIMERE_TYPE_Q6_K: return (wbits & 1) ? cudaErrorInvalidValue : go(kquant_mmvq_kernel<CHIMERE_TYPE_Q6_K>);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_mmvq_kquant(int wtype, const void* w, const void* xq8, float* y, int ncols, int nrows, cudaStream_t stream) {
    return launch_mmvq_kquant_batched(wtype, w, nullptr, xq8, 0, y, nullptr, 0, 1, ncols, nrows, 0, nullptr, true, stream);
}

cudaError_t launch_act_q8_1(const float* g, const float* u, int64_t in_stride, void* out, int64_t out_stride, int T, int F, cudaStream_t stream) {
    if (T <= 0 || F <= 0) return cudaSuccess;
    if (F & 31) return cudaErrorInvalidValue;
    const int64_t warps = (int64_t)T * (F >> 5);
    return launch_pdl(act_q8_1_kernel, dim3((unsigned)((warps + 7) / 8)), 256, 0, stream, g, u, in_stride, (uint8_t*)out, out_stride, T, F);
}

}  // namespace chimere
