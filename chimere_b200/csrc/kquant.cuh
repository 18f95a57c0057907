// kquant.cuh -- a 32-weight sub-block of a K-quant row in registers, and its product with a Q8_1 block.
#pragma once
#include "common.cuh"

namespace chimere {

__device__ __forceinline__ uint32_t ld32(const uint8_t* p) { return *reinterpret_cast<const uint32_t*>(p); }

// six-bit scale and min of sub-block j from the twelve packed bytes (ffi/src/lib.rs:368-383)
__device__ __forceinline__ void scale_min_k4(int j, const uint8_t* sc, int& s, int& m) {
    if (j < 4) { s = sc[j] & 63; m = sc[j + 4] & 63; }
    else { s = (sc[j + 4] & 0x0F) | ((sc[j - 4] >> 6) << 4); m = (sc[j + 4] >> 4) | ((sc[j] >> 6) << 4); }
}

template <int TYPE> struct KBlock;
template <> struct KBlock<CHIMERE_TYPE_Q4_K> { static constexpr int kBytes = 144, kQs = 16; };
template <> struct KBlock<CHIMERE_TYPE_Q5_K> { static constexpr int kBytes = 176, kQs = 48; };
template <> struct KBlock<CHIMERE_TYPE_Q6_K> { static constexpr int kBytes = 210, kQs = 0; };

// A decoded 32-weight sub-block: eight words of four quants each and what scales them.
struct SubBlock {
    int w[8];
    float d, dmin;   // super-block scales (dmin unused for Q6_K)
    int sc, mn;      // Q4_K / Q5_K: six-bit scale and min; Q6_K: the int8 scales of the first and the second 16 weights
};

template <int TYPE>
__device__ __forceinline__ void decode_sub(const uint8_t* blk, int j, SubBlock& s) {
    if (TYPE == CHIMERE_TYPE_Q6_K) {
        // 210-byte blocks are only 2-byte aligned
        const int grp = j >> 2, q = j & 3;
        const uint8_t* ql = blk + 64 * grp + 32 * (q & 1);
        const uint8_t* qh = blk + 128 + 32 * grp;
        const int8_t* sc = reinterpret_cast<const int8_t*>(blk + 192) + 8 * grp + 2 * q;
        s.d = h2f(ld_u16(blk + 208)); s.dmin = 0.0f;
        s.sc = sc[0]; s.mn = sc[1];
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            const uint32_t lo = ld_u32_a2(ql + 4 * g), hi = ld_u32_a2(qh + 4 * g);
            const uint32_t nib = (q >> 1) ? (lo >> 4) & 0x0F0F0F0Fu : lo & 0x0F0F0F0Fu;
            const uint32_t v = nib | (((hi >> (2 * q)) & 0x03030303u) << 4);      // 0..63 per byte
            s.w[g] = (int)__vsub4(v, 0x20202020u);                                // -32..31 per byte
        }
    } else {
        s.d = h2f(ld_u16(blk)); s.dmin = h2f(ld_u16(blk + 2));
        scale_min_k4(j, blk + 4, s.sc, s.mn);
        const uint8_t* qs = blk + KBlock<TYPE>::kQs + 32 * (j >> 1);
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            const uint32_t lo = ld32(qs + 4 * g);
            uint32_t v = (j & 1) ? (lo >> 4) & 0x0F0F0F0Fu : lo & 0x0F0F0F0Fu;
            if (TYPE == CHIMERE_TYPE_Q5_K) v |= ((ld32(blk + 16 + 4 * g) >> j) & 0x01010101u) << 4;
            s.w[g] = (int)v;
        }
    }
}

// acc + its product with one Q8_1 block `xb` (36 bytes: f16 d, f16 s, 32 int8).  The rounding is written out, addition included: a row has the
// same bits in every kernel, whatever the compiler would make of a product and a sum there.
template <int TYPE>
__device__ __forceinline__ float add_dot(float acc, const SubBlock& s, const uint8_t* xb) {
    const __half2 ds = *reinterpret_cast<const __half2*>(xb);
    const float d8 = __low2float(ds), s8 = __high2float(ds);
    if (TYPE == CHIMERE_TYPE_Q6_K) {
        int da = 0, db = 0;
#pragma unroll
        for (int g = 0; g < 4; ++g) { da = __dp4a(s.w[g], (int)ld32(xb + 4 + 4 * g), da); db = __dp4a(s.w[4 + g], (int)ld32(xb + 20 + 4 * g), db); }
        return fmaf(__fmul_rn(s.d, d8), (float)(s.sc * da + s.mn * db), acc);
    } else {
        int dot = 0;
#pragma unroll
        for (int g = 0; g < 8; ++g) dot = __dp4a(s.w[g], (int)ld32(xb + 4 + 4 * g), dot);
        return __fadd_rn(acc, fmaf(-__fmul_rn(s.dmin, (float)s.mn), s8, __fmul_rn(__fmul_rn(s.d, d8), (float)(s.sc * dot))));
    }
}

// The same with the type known at run time (the shared expert beside the routed experts' kernels, pairs.cu).
__device__ __forceinline__ int kquant_block_bytes(int type) {
    return type == CHIMERE_TYPE_Q4_K ? KBlock<CHIMERE_TYPE_Q4_K>::kBytes : type == CHIMERE_TYPE_Q5_K ? KBlock<CHIMERE_TYPE_Q5_K>::kBytes : KBlock<CHIMERE_TYPE_Q6_K>::kBytes;
}
__device__ __forceinline__ void decode_sub(int type, const uint8_t* row, int sb, SubBlock& s) {
    const uint8_t* blk = row + (size_t)(sb >> 3) * kquant_block_bytes(type);
    if (type == CHIMERE_TYPE_Q5_K) decode_sub<CHIMERE_TYPE_Q5_K>(blk, sb & 7, s);
    else if (type == CHIMERE_TYPE_Q4_K) decode_sub<CHIMERE_TYPE_Q4_K>(blk, sb & 7, s);
    else decode_sub<CHIMERE_TYPE_Q6_K>(blk, sb & 7, s);
}
__device__ __forceinline__ float add_dot(int type, float acc, const SubBlock& s, const uint8_t* xb) {
    return type == CHIMERE_TYPE_Q6_K ? add_dot<CHIMERE_TYPE_Q6_K>(acc, s, xb) : add_dot<CHIMERE_TYPE_Q5_K>(acc, s, xb);   // (Q4_K: as Q5_K)
}

}  // namespace chimere
