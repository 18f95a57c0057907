// common.cuh -- device helpers shared by the MoE kernels (sm_100a only).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/chimere_b200_moe.h"

#if defined(__CUDA_ARCH__) && (__CUDA_ARCH__ < 1000)
#error "this library is written for sm_100a only"
#endif

namespace chimere {

constexpr int kQ81Bytes = 36;
constexpr int kMaxGroupTokens = 8;   // tokens one GEMV work entry carries
constexpr int kSharedGroupTokens = 2;  // ... for the shared expert (every token uses it): smaller entries balance the grid
// Decode-size batches give every token its own shared-expert entry: the kernels stage one token per pass there, and
// a second pass in the same CTA is a longer chain than a second CTA reading the shared matrices from L2.
constexpr int kSingleSharedTokens = 8;
__host__ __device__ inline int shared_group_tokens(int T) { return T <= kSingleSharedTokens ? 1 : kSharedGroupTokens; }
// Tokens per routed entry.  In a decode-size batch every pair is an entry of its own: a popular expert's pairs are spread over
// the SMs (its matrices then come from L2 again) instead of being a chain of passes in one CTA -- 8 skewed tokens through 256
// Q4_0 experts of 512 x 2048 63 -> 35 us, 8 uniform ones 58 -> 38.  Matrices of more than 2M weights (1856 x 2688) cost more to fetch
// twice than a second pass: two pairs per entry.  `wide`: Q8_0 matrices (139 KB of gate and up rows in a CTA, one CTA per SM) do
// so at any size -- 8 skewed tokens take 78 us in entries of up to eight pairs and 117 in entries of one, 24 tokens 124 and 295 -- and
// so do the kernels on raw ggml blocks, which unpack a row once per entry (Q4_0, 8 / 24 skewed tokens 81 / 134 us and 91 / 227).
constexpr int kFewTokens = 40;   // the largest batch for which the GEMV kernels are sized for one or two pairs per expert
constexpr int kSinglePairTokens = 24;   // ... and for one
constexpr int kFewTokensWide = 16;      // Q8_0: the largest batch for which they are sized for as many CTAs as one token per pass allows
__host__ __device__ inline int group_tokens(int T, int64_t weights, bool wide) {
    return wide || T > kFewTokens ? kMaxGroupTokens : weights > (1 << 21) || T > kSinglePairTokens ? 2 : 1;
}
// Behind each of these batch sizes the entries get longer and their number can fall: a work list is sized for every one below its capacity.
constexpr int kEntrySteps[] = {kSingleSharedTokens, kSinglePairTokens, kFewTokens};
constexpr int kMaxTopK = 8;
constexpr int kMaxExperts = 256;

// Work list the routing kernel leaves for the grouped GEMV kernels: word 0 = number of entries, word 1 = routed
// entries, word 2 = shared-expert entries; entries start at word 4, kListEntry words each:
// { expert id (-1 = shared expert), start, m, 0, pair row of token 0 .. 7 }.  Routed entry: pairs
// perm[start .. start+m) (the pair rows repeat them so a kernel needs no second look-up); shared entry:
// tokens start .. start+m, pair rows T*top_k + token.  The shared expert's entries come first: they carry the
// most tokens and should start early.
constexpr int kListHeader = 4;
constexpr int kListEntry = 12;

// status bits a kernel may raise in the workspace status word
constexpr int kStatusWaitTimeout = 1;
constexpr int kStatusListFull = 2;

__device__ __forceinline__ float h2f(uint32_t bits) { return __half2float(__ushort_as_half((unsigned short)bits)); }
__device__ __forceinline__ uint32_t ld_u16(const uint8_t* p) { return *reinterpret_cast<const uint16_t*>(p); }
// 32-bit load from an address that is only 2-byte aligned (ggml blocks are 2-byte aligned).
__device__ __forceinline__ uint32_t ld_u32_a2(const uint8_t* p) { return ld_u16(p) | (ld_u16(p + 2) << 16); }

// PTX prmt in its default mode: selector nibble bit 3 replicates the sign bit of the chosen byte.
// (__byte_perm documents only the low three selector bits, so the instruction is spelled out.)
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- mbarrier + bulk async copy (global -> shared), no multicast -------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cta(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// dst and src 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
// Bounded wait on phase `parity`; false if the limit ran out (caller raises a status bit).  A try that finds the phase incomplete comes
// back after 7770 cycles (4 us), so the limit is about a second.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok = 0;
    for (int it = 0; it < (1 << 18) && !ok; ++it) {
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    }
    return ok != 0;
}

// ---- two fp32 lanes in one 64-bit register (sm_100 has two-wide fp32 add / mul / fma, each lane rounded like the scalar form) ----
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi)); return r; }
__device__ __forceinline__ uint64_t pack2f(float lo, float hi) { return pack2(__float_as_uint(lo), __float_as_uint(hi)); }
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) { uint64_t d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) { uint64_t d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }

// Counter increment that publishes this thread's (and, behind a CTA barrier, its CTA's) earlier writes and makes the
// writes published by the other arrivals visible: release and acquire in the one instruction, instead of a fence on
// either side of a relaxed atomic.  Returns the old value.
__device__ __forceinline__ int atom_add_acq_rel_gpu(int* p, int v) {
    int old;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

// ---- programmatic dependent launch ---------------------------------------------------------
// A kernel launched with the programmatic-serialization attribute may start while its predecessor in the
// stream still runs; griddep_wait() blocks until that predecessor has completed and its writes are visible
// (a no-op for a normally launched kernel).  griddep_launch() lets the successor's CTAs start once every CTA
// of this grid has called it or exited.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---- per-type decode of one 32-weight unit into eight int8x4 words -----------------------
// Unit b of a row = 32 consecutive weights (a Q4_0 / Q8_0 block, or sub-block b%8 of IQ3_S
// super-block b/8).  load() returns the signed int8 weights packed four per word such that
// finish(sum_g dp4a(w[g], q8word[g]), mul) is the integer block dot (Q4_0 words carry 16x the weight,
// IQ3_S units a per-sub-block multiplier `mul`).
template <int TYPE> struct Unit;

template <> struct Unit<CHIMERE_TYPE_Q8_0> {
    static constexpr int kBlockBytes = 34, kBlockElems = 32;
    __device__ static __forceinline__ int64_t row_bytes(int ncols) { return (int64_t)(ncols >> 5) * 34; }
    __device__ static __forceinline__ void load(const uint8_t* row, int b, const uint32_t*, int (&w)[8], float& dw, int& mul) {
        const uint8_t* blk = row + b * 34;
        dw = h2f(ld_u16(blk));
        mul = 1;
#pragma unroll
        for (int g = 0; g < 8; ++g) w[g] = (int)ld_u32_a2(blk + 2 + 4 * g);
    }
    __device__ static __forceinline__ int finish(int sumi, int mul) { (void)mul; return sumi; }
};

template <> struct Unit<CHIMERE_TYPE_Q4_0> {
    static constexpr int kBlockBytes = 18, kBlockElems = 32;
    __device__ static __forceinline__ int64_t row_bytes(int ncols) { return (int64_t)(ncols >> 5) * 18; }
    // byte = ((nibble ^ 8) << 4) read as int8 = 16 * (nibble - 8); the dot comes out times 16.
    __device__ static __forceinline__ void load(const uint8_t* row, int b, const uint32_t*, int (&w)[8], float& dw, int& mul) {
        const uint8_t* blk = row + b * 18;
        dw = h2f(ld_u16(blk));
        mul = 1;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            uint32_t t = ld_u32_a2(blk + 2 + 4 * j) ^ 0x88888888u;
            w[j] = (int)((t << 4) & 0xF0F0F0F0u);   // low nibbles: elements 4j .. 4j+3
            w[4 + j] = (int)(t & 0xF0F0F0F0u);      // high nibbles: elements 16+4j ..
        }
    }
    __device__ static __forceinline__ int finish(int sumi, int mul) { (void)mul; return sumi >> 4; }
};

template <> struct Unit<CHIMERE_TYPE_IQ3_S> {
    static constexpr int kBlockBytes = 110, kBlockElems = 256;
    __device__ static __forceinline__ int64_t row_bytes(int ncols) { return (int64_t)(ncols >> 8) * 110; }
    // Layout of the 110-byte super-block: d f16 @0, qs[64] @2, qh[8] @66, signs[32] @74, scales[4] @106.
    __device__ static __forceinline__ void load(const uint8_t* row, int b, const uint32_t* grid, int (&w)[8], float& dw, int& mul) {
        const uint8_t* blk = row + (b >> 3) * 110;
        const int sg = b & 7;
        dw = h2f(ld_u16(blk));
        const uint32_t q0 = ld_u32_a2(blk + 2 + sg * 8), q1 = ld_u32_a2(blk + 6 + sg * 8);
        const uint32_t qh = blk[66 + sg];
        const uint32_t sgn = ld_u32_a2(blk + 74 + sg * 4);
        const uint32_t scb = blk[106 + (sg >> 1)];
        mul = 1 + 2 * (int)((scb >> ((sg & 1) * 4)) & 15u);
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            const uint32_t qsb = ((g < 4 ? q0 : q1) >> (8 * (g & 3))) & 0xFFu;
            const uint32_t gv = grid[qsb | (((qh >> g) & 1u) << 8)];
            // 4 sign bits -> bit 7 of each byte -> 0xFF/0x00 byte mask; -m = (m ^ 0xFF) + 1 never
            // carries out of its byte because every magnitude is >= 1.
            const uint32_t t7 = (((sgn >> (4 * g)) & 15u) * 0x10204080u) & 0x80808080u;
            const uint32_t mask = prmt(t7, 0u, 0xBA98u);
            w[g] = (int)((gv ^ mask) + (t7 >> 7));
        }
    }
    __device__ static __forceinline__ int finish(int sumi, int mul) { return sumi * mul; }
};

template <int TYPE>
__device__ __forceinline__ int unit_sumi(const int (&w)[8], int mul, const int* q8words) {
    int s = 0;
#pragma unroll
    for (int g = 0; g < 8; ++g) s = __dp4a(w[g], q8words[g], s);
    return Unit<TYPE>::finish(s, mul);
}

// Sum of 256 partials held in shared memory in the order of a binary tree with strides
// 128, 64, ..., 1 (element i+stride added into element i), done by one warp.
__device__ __forceinline__ float tree256(const float* r, int lane) {
    float a0 = r[lane] + r[lane + 128];
    float a1 = r[lane + 32] + r[lane + 160];
    float a2 = r[lane + 64] + r[lane + 192];
    float a3 = r[lane + 96] + r[lane + 224];
    float b0 = a0 + a2;
    float b1 = a1 + a3;
    float v = b0 + b1;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) v += __shfl_down_sync(0xffffffffu, v, s);
    return v;  // valid in lane 0
}

// Sigmoid and SiLU exactly as the reference spells them (chimere_kernels.cu:1545, scratch_pool.rs:272).
__device__ __forceinline__ float sigmoid_ref(float v) { return 1.0f / (1.0f + expf(-v)); }
__device__ __forceinline__ float silu_mul_ref(float g, float u) { float s = g / (1.0f + expf(-g)); return s * u; }
// The same for the kernel that stands on the instructions of this step (T = 8192, Q8_0, skewed routing: 1980 us with the division
// operator, 1942 with this): the quotient from the hardware's reciprocal estimate and one correction by the remainder (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", 1990).  For every g above -87 the bits are those of
// silu_mul_ref (compared over all 2^32 values, infinities and NaN among them; only -0 gives +0).  Below, where the estimate leaves the normal
// numbers, it lies between -2.5e-36 and 0 (the exact one between -1.2e-36 and 0), and -88.8 and less give -0 as there.
__device__ __forceinline__ float silu_mul_fast(float g, float u) {
    const float b = 1.0f + expf(-g);
    float r, s;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(b));
    s = g * r;
    s = fmaf(fmaf(-s, fminf(b, 8.5070592e37f), g), r, s);   // (2^126: no infinity in the remainder)
    return (g > 64.0f ? g : s) * u;   // (the denominator is 1 there; infinity has no remainder)
}
// roundf(x) as an integer, |x| < 2^22: half away from zero.  (The addition rounds towards zero, so that 0.5 - 2^-25 stays below 1.)
__device__ __forceinline__ int round_int(float x) { return __float2int_rz(__fadd_rz(x, copysignf(0.5f, x))); }

// One 32-value block of Q8_1 by one warp, lane = value: d = amax / 127 and q = roundf(v / d), both quotients correctly rounded as
// the division operator's are: with the correctly rounded reciprocal r of b, the last of
//   q0 = a * r,  q1 = q0 + r * (a - b * q0),  q2 = q1 + r * (a - b * q1)
// is the correctly rounded a / b (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990,
// theorem on division by a correctly rounded reciprocal) as long as nothing underflows or overflows.  Blocks outside a wide
// range of magnitudes, and blocks with a NaN, which the maximum leaves out, take the plain operations.
__device__ __forceinline__ float div_by_recip(float a, float b, float r) {
    float q = a * r;
    q = fmaf(fmaf(-q, b, a), r, q);
    return fmaf(fmaf(-q, b, a), r, q);
}
__device__ __forceinline__ int8_t q8_1_warp(float v, float& d) {
    // largest magnitude: bit patterns of non-negative floats order like the values, with the NaNs above infinity
    float amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(v))));
    if (amax > 1e-25f && amax < 1e25f) {
        d = div_by_recip(amax, 127.0f, 1.0f / 127.0f);
        return (int8_t)round_int(div_by_recip(v, d, __frcp_rn(d)));
    }
    amax = fabsf(v);
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, s));
    d = amax / 127.0f;
    return amax == 0.0f ? (int8_t)0 : (int8_t)roundf(v / d);
}

}  // namespace chimere
