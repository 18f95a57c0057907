// pairs.cu -- decode batches on tiled32 weights: every (token, expert) pair is a work item of its own and needs no work list.
//
// The two expert launches of a layer take their experts straight from the router's logits: each CTA repeats the top-k of the tokens
// that its items belong to, which is shorter than waiting for one CTA at the router's end to do it for all, sort the pairs and write
// a list.  The sorted order (perm, offsets, the list) is still left in the workspace, by a CTA of the down launch beside the others.
//
//   pair_gate_up_kernel : item = (pair or shared-expert token, 32-row tile); a CTA's warps are the K slices of the tile.  Weights go
//                         from global memory to registers, a group of four units ahead (every unit's registers are asked for
//                         again, for a later group or the CTA's next item, as soon as it is decoded), so there is always a
//                         CTA's worth of loads in flight and no staging, barrier or copy to issue between them.
//   pair_down_kernel    : item = (token, 32-row tile); the CTA holds a warp (or several, by K slices) for every one of the token's
//                         experts, so the combine is a sum over shared memory: no per-pair rows to read back, no counters.
//                         Started behind the gate/up launch, it looks up its experts and has its first weights in flight
//                         before that launch ends.
//
// Sums are bit for bit those of bulk_kernel (gemv_tiled.cu): same K slices, same order.
//
// What bounds it.  One to two tokens: three chains per layer (256 IQ3_S / Q4_0 experts, H 2048, F 512, one token, us: router 0.7 behind the wait, logits to
// experts 1.6 - 2.5, weights and products 2.0, a grid's end to the next one's start 0.8 each time, down stage 3.1).  From eight tokens on the weights'
// latency under the same chains: with 15 warps per SM (registers) gate/up asks for enough to keep DRAM 41 % busy, down 23 %, and 47 and 37 % of
// the issue slots are used (captured alone, cold).  Layer, us, against the list and bulk_kernel with its one item per CTA and 7 400 warp instructions per item (here 4 000):
// 1 token 18.1 -> 13.4, 2: 21.6 -> 15.4, 5: 29.8 -> 23.0, 8: 38.3 -> 30.7, 16: 57.3 -> 47.6, 24: 77.8 -> 65.1.
#include "common.cuh"
#include "kernels.h"
#include "kquant.cuh"
#include "routing.cuh"
#include "tiled.cuh"

namespace chimere {

constexpr int kPairItems = 64;      // items of a CTA (their experts are looked up together)

// (a predicated weight load, as those of tiled.cuh)
__device__ __forceinline__ void ldg128_if(uint4& v, const uint8_t* a, int on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t@p ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
                 : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w) : "l"(a), "r"(on));
}
__device__ __forceinline__ void sts_v4(uint32_t a, const uint4& v) { asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory"); }
__device__ __forceinline__ void sts_v2(uint32_t a, uint32_t x, uint32_t y) { asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(x), "r"(y) : "memory"); }

// Four units of a lane's row, in registers.  dot16 = 16 * sl + sh (see Tiled<>::finish) is 16 times the block dot of Q4_0 and 8 times
// that of IQ3_S without its sub-block factor; the power of two comes out of the weight scale, which is exact.
template <int TYPE> struct PairGroup;
template <> struct PairGroup<CHIMERE_TYPE_Q4_0> {
    uint4 v[4];
    uint16_t d[4];
    // gp: the group's first byte + 16 * lane (at()); offsets from there are constants, but for the scales' -14 * lane
    __device__ static __forceinline__ const uint8_t* at(const uint8_t* tile, int g, int lane) { return tile + (uint32_t)(g * 2304 + lane * 16); }
    __device__ __forceinline__ void load_unit(int u, const uint8_t* gp, int lane, int on) {
        ldg128_if(v[u], gp + u * 576, on);
        ldg16_if(d[u], gp - lane * 14 + (u * 576 + 512), on);
    }
    __device__ __forceinline__ void load_scales(const uint8_t*, int, int, int) {}
};
template <> struct PairGroup<CHIMERE_TYPE_IQ3_S> {
    uint4 v[4];
    uint16_t d;
    uint32_t sc;
    __device__ static __forceinline__ const uint8_t* at(const uint8_t* tile, int g, int lane) { return tile + (uint32_t)((g >> 1) * 4288 + (g & 1) * 2048 + lane * 16); }
    __device__ __forceinline__ void load_unit(int u, const uint8_t* gp, int lane, int on) { ldg128_if(v[u], gp + u * 512, on); }
    __device__ __forceinline__ void load_scales(const uint8_t* gp, int g, int lane, int on) {
        const uint8_t* a = gp + (4096 - (g & 1) * 2048) - lane * 14;
        ldg16_if(d, a, on);
        ldg32_if(sc, a + 64 + lane * 2, on);
    }
};
template <int TYPE>
__device__ __forceinline__ void fill_group(PairGroup<TYPE>& r, const uint8_t* tile, int g, int lane, int nu) {
    const uint8_t* gp = PairGroup<TYPE>::at(tile, g, lane);
#pragma unroll
    for (int u = 0; u < kGroupUnits; ++u) r.load_unit(u, gp, lane, u < nu);
    r.load_scales(gp, g, lane, nu > 0);
}

__device__ __forceinline__ int dot16(const uint4& v, const uint4& q0, const uint4& q1, int corr, bool corr_low) {
    const uint32_t x[4] = {v.x, v.y, v.z, v.w};
    const int a[4] = {(int)q0.x, (int)q0.y, (int)q0.z, (int)q0.w}, b[4] = {(int)q1.x, (int)q1.y, (int)q1.z, (int)q1.w};
    int sl = corr_low ? corr : 0, sh = corr_low ? 0 : corr;
#pragma unroll
    for (int j = 0; j < 4; ++j) { sl = dp4a_us(x[j] & 0x0F0F0F0Fu, a[j], sl); sh = __dp4a((int)(x[j] & 0xF0F0F0F0u), b[j], sh); }
    return 16 * sl + sh;
}

// One group of one or two matrices against the token at shared addresses xq (int8 plane) / xd ({ f32 scale, correction word } per
// unit), both of the group's first unit; nu units.  The registers are asked for again from group gn of tiles na / nb (nn units there).
// AHEAD: a unit's token values are loaded in front of the products of the unit before (a warp issues in order), where there are registers
// for that: ungated experts of 1856 columns, 12 tokens, four layers 466 -> 441 us (and 416 with three groups of a down row in flight instead of
// four, which spilled 108 bytes); gated ones and short down rows gain nothing.
template <int TYPE, bool DUAL, bool AHEAD>
__device__ __forceinline__ void pair_group(PairGroup<TYPE>& ra, PairGroup<TYPE>& rb, int g, int nu, uint32_t xq, uint32_t xd, float& acc_a, float& acc_b,
                                           const uint8_t* na, const uint8_t* nb, int gn, int nn, int lane) {
    constexpr bool kLow = Tiled<TYPE>::kCorrLow, kGroupScale = Tiled<TYPE>::kGroupScale;
    const uint8_t* pna = PairGroup<TYPE>::at(na, gn, lane);
    const uint8_t* pnb = DUAL ? PairGroup<TYPE>::at(nb, gn, lane) : nullptr;
    float pa = 0.0f, pb = 0.0f;
    uint32_t sa = 0, sb = 0;
    if constexpr (TYPE == CHIMERE_TYPE_IQ3_S) { sa = ra.sc >> (16 * (g & 1)); if (DUAL) sb = rb.sc >> (16 * (g & 1)); }
    uint4 q0[2], q1[2];
    uint2 dc[2];
    auto token = [&](int u) { q0[u & 1] = lds128(xq + u * 32); q1[u & 1] = lds128(xq + u * 32 + 16); dc[u & 1] = lds64(xd + u * 8); };
    if (AHEAD) token(0);
#pragma unroll
    for (int u = 0; u < kGroupUnits; ++u) {
        if (AHEAD ? u + 1 < kGroupUnits : u < nu) token(AHEAD ? u + 1 : u);
        if (u < nu) {
            const float dx = __uint_as_float(dc[u & 1].x);
            const int corr = (int)dc[u & 1].y;
            int ta = dot16(ra.v[u], q0[u & 1], q1[u & 1], corr, kLow), tb = DUAL ? dot16(rb.v[u], q0[u & 1], q1[u & 1], corr, kLow) : 0;
            if constexpr (TYPE == CHIMERE_TYPE_IQ3_S) {
                ta *= (int)(1u + 2u * ((sa >> (4 * u)) & 15u));
                pa = fmaf((float)ta, dx, pa);
                if (DUAL) { tb *= (int)(1u + 2u * ((sb >> (4 * u)) & 15u)); pb = fmaf((float)tb, dx, pb); }
            } else {
                acc_a = fmaf(h2f(ra.d[u]) * 0.0625f * dx, (float)ta, acc_a);
                if (DUAL) acc_b = fmaf(h2f(rb.d[u]) * 0.0625f * dx, (float)tb, acc_b);
            }
        }
        ra.load_unit(u, pna, lane, u < nn);
        if (DUAL) rb.load_unit(u, pnb, lane, u < nn);
    }
    if constexpr (kGroupScale) {
        acc_a = fmaf(h2f(ra.d) * 0.125f, pa, acc_a);
        if (DUAL) acc_b = fmaf(h2f(rb.d) * 0.125f, pb, acc_b);
    }
    ra.load_scales(pna, gn, lane, nn > 0);
    if (DUAL) rb.load_scales(pnb, gn, lane, nn > 0);
}

// A warp's part of a token's Q8_1 planes: lane = unit (at most 32 units), on its way to the warp's own shared memory.
struct PairX { uint4 a, b; float d; };
__device__ __forceinline__ void load_x(PairX& x, const GemvParams& p, int row, int u0, int nu, int lane) {
    if (lane < nu) {
        const uint4* q = reinterpret_cast<const uint4*>(p.in_soa_q + (size_t)row * p.in_soa_q_stride + (u0 + lane) * 32);
        x.a = __ldcg(q); x.b = __ldcg(q + 1);
        x.d = __ldcg(p.in_soa_d + (size_t)row * p.in_soa_d_stride + u0 + lane);
    }
}
template <int TYPE>
__device__ __forceinline__ void store_x(uint32_t xq, uint32_t xd, const PairX& x, int nu, int lane) {
    __syncwarp();   // (every lane has read what was there)
    if (lane < nu) {
        sts_v4(xq + lane * 32, x.a);
        sts_v4(xq + lane * 32 + 16, x.b);
        sts_v2(xd + lane * 8, __float_as_uint(x.d), (uint32_t)Tiled<TYPE>::correction(sum16(x.a), sum16(x.b)));
    }
    __syncwarp();
}

// grid: any number of CTAs (an item list dealt round); block = 32 * (K slices).  upw = units per slice.
// KQ: a K-quant shared expert's up and gate rows ride along, a row per warp of those that have no top-k to do first (its weights
// are asked for before the router has ended); its activation is the down launch's.  Three launches of its own behind the layer otherwise:
// half-layer of two tokens 32 us with them, 20 with the rows here and the norm in the router.
constexpr int kKqSub = 2;   // sub-blocks of a row per lane: H <= 2048
template <int TYPE, bool DUAL, bool KQ, int D, int CTAS>
__global__ void __launch_bounds__(256, CTAS) pair_gate_up_kernel(const __grid_constant__ RouteParams r, const __grid_constant__ GemvParams p,
                                                                 const __grid_constant__ PairExtras x, int upw) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ int4 s_item[kPairItems];   // { output row, token, row tile, expert or -1 = shared }
    constexpr int kMat = DUAL ? 2 : 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wk = blockDim.x >> 5;
    const int T = p.T, k = p.top_k, P = T * k, tiles_s = p.nrows_shared >> 5, n_sh = T * tiles_s, n_items = n_sh + P * (p.nrows_routed >> 5);
    const int ni = max(0, (n_items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x);
    const int nb = p.H >> 5, u0 = min(nb, warp * upw), nu_x = min(nb, u0 + upw) - u0, g0 = u0 >> 2, ng = nu_x >> 2;   // (H is a multiple of 128)
    const uint32_t xq = smem_u32(smem) + (uint32_t)(warp * upw * 40), xd = xq + (uint32_t)upw * 32;
    float* red = reinterpret_cast<float*>(smem + (size_t)wk * upw * 40);   // [2][matrix][slice][32]

    // consecutive items share a row tile: the shared expert's matrices, and experts that several tokens chose, come from L2
    auto item = [&](int n) {
        if (n < n_sh) { const int tile = n / T, t = n - tile * T; return make_int4(P + t, t, tile, -1); }
        const int m = n - n_sh, tile = m / P, q = m - tile * P;
        return make_int4(q, q / k, tile, 0);
    };
    for (int i = tid; i < ni; i += blockDim.x) s_item[i] = item((int)blockIdx.x + i * (int)gridDim.x);
    const int first_token = ni > 0 ? item((int)blockIdx.x).y : 0;
    // the K-quant rows of warps 1 ..
    const int kq_warps = (int)gridDim.x * (wk - 1), kq_rows = KQ ? 2 * x.F_s : 0;
    int kq = (int)blockIdx.x * (wk - 1) + warp - 1;
    SubBlock ks[kKqSub];
    auto kq_load = [&]() {
        const bool gate = kq >= x.F_s;
        const uint8_t* row = (gate ? x.gate : x.up) + (size_t)(gate ? kq - x.F_s : kq) * (size_t)((p.H >> 8) * kquant_block_bytes(x.type));
#pragma unroll
        for (int i = 0; i < kKqSub; ++i)
            if (lane + 32 * i < nb) decode_sub(x.type, row, lane + 32 * i, ks[i]);
    };
    if (KQ && warp > 0 && kq < kq_rows) kq_load();
    griddep_wait();
    if (tid == 0) griddep_launch();
    PairX xr;
    load_x(xr, p, first_token, u0, nu_x, lane);
    if (x.hidden)   // the half-layer's residual: the router has read the old one
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + tid; i < (int64_t)T * p.H; i += (int64_t)gridDim.x * blockDim.x) x.residual[i] = x.hidden[i] + x.residual[i];
    __syncthreads();
    for (int i = warp; i < ni; i += wk) {
        const int4 it = s_item[i];
        if (it.w >= 0) {
            const int slot = it.x - it.y * k;
            const TopkSlot s = topk_select(r, r.router_logits + (size_t)it.y * r.E, lane, slot + 1);
            if (lane == slot) s_item[i].w = s.id;
        }
    }
    if (KQ && warp > 0) {
        while (kq < kq_rows) {
            const bool gate = kq >= x.F_s;
            float* out = x.rows + (gate ? (size_t)T * x.F_s + kq - x.F_s : (size_t)kq);
            for (int t0 = 0; t0 < T; t0 += 4) {   // (kquant_mmvq_kernel's order: a lane's sub-blocks in sequence, then the lanes in a butterfly)
                float v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    v[j] = 0.0f;
                    const uint8_t* xb = p.in_q8 + (size_t)min(t0 + j, T - 1) * p.in_stride + (size_t)lane * kQ81Bytes;
#pragma unroll
                    for (int i = 0; i < kKqSub; ++i)
                        if (lane + 32 * i < nb) v[j] = add_dot(x.type, v[j], ks[i], xb + i * 32 * kQ81Bytes);
                }
#pragma unroll
                for (int s = 16; s > 0; s >>= 1)
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[j] += __shfl_xor_sync(0xffffffffu, v[j], s);
                if (lane == 0)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (t0 + j < T) out[(size_t)(t0 + j) * x.F_s] = v[j];
            }
            kq += kq_warps;
            if (kq < kq_rows) kq_load();
        }
    }
    __syncthreads();
    if (ni == 0) return;

    const int64_t tb = Tiled<TYPE>::tile_bytes(p.H);
    auto up_tile = [&](const int4& it) { return (it.w < 0 ? p.sh_b : p.w_b + (size_t)it.w * p.stride_b) + (size_t)it.z * tb; };
    auto gate_tile = [&](const int4& it) { return DUAL ? (it.w < 0 ? p.sh_a : p.w_a + (size_t)it.w * p.stride_a) + (size_t)it.z * tb : nullptr; };
    PairGroup<TYPE> ra[D], rb[D];   // up, gate
    int4 it = s_item[0];
    const uint8_t* ta = up_tile(it);
    const uint8_t* tg = gate_tile(it);
#pragma unroll
    for (int d = 0; d < D; ++d) {
        fill_group<TYPE>(ra[d], ta, g0 + d, lane, d < ng ? 4 : 0);
        if (DUAL) fill_group<TYPE>(rb[d], tg, g0 + d, lane, d < ng ? 4 : 0);
    }
    for (int i = 0; i < ni; ++i) {
        const bool more = i + 1 < ni;
        const int4 nx = s_item[more ? i + 1 : i];
        const uint8_t* na = up_tile(nx);
        const uint8_t* ngt = gate_tile(nx);
        store_x<TYPE>(xq, xd, xr, nu_x, lane);
        if (more) load_x(xr, p, nx.y, u0, nu_x, lane);
        float acc_u = 0.0f, acc_g = 0.0f;
        for (int gg = 0; gg < ng; gg += D) {
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const int g = gg + d;
                if (g < ng) {
                    const bool same = g + D < ng;
                    pair_group<TYPE, DUAL, true>(ra[d], rb[d], g0 + g, 4, xq + (uint32_t)g * 128, xd + (uint32_t)g * 32, acc_u, acc_g, same ? ta : na, same ? tg : ngt,
                                           g0 + (same ? g + D : d), same || more ? 4 : 0, lane);
                }
            }
        }
        float* mine = red + (i & 1) * (kMat * wk * 32);
        mine[warp * 32 + lane] = acc_u;
        if (DUAL) mine[(wk + warp) * 32 + lane] = acc_g;
        __syncthreads();   // (the other half of `red` is free again: its reader has come to this barrier too)
        if (warp == i % wk) {
            // sum of the K slices, activation, Q8_1 of the 32 results (lane = element)
            float u = 0.0f, g = 0.0f;
            for (int s = 0; s < wk; ++s) {
                u += mine[s * 32 + lane];
                if (DUAL) g += mine[(wk + s) * 32 + lane];
            }
            float v;
            if (DUAL) v = silu_mul_ref(g, u);
            else { const float a = fmaxf(u, 0.0f); v = a * a; }
            float sum = v;
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
            float d;
            const int8_t q = q8_1_warp(v, d);
            uint8_t* out = p.inter_q8 + (size_t)it.x * p.inter_stride + (size_t)it.z * kQ81Bytes;
            reinterpret_cast<int8_t*>(out)[4 + lane] = q;
            p.out_soa_q[(size_t)it.x * p.out_soa_q_stride + (size_t)it.z * 32 + lane] = q;
            if (lane == 0) {
                const __half dh = __float2half(d);
                *reinterpret_cast<__half2*>(out) = __halves2half2(dh, __float2half(sum));
                p.out_soa_d[(size_t)it.x * p.out_soa_d_stride + it.z] = __half2float(dh);
            }
        }
        it = nx; ta = na; tg = ngt;
    }
}

// How the down launch deals the K slices of a token's experts to warps.
struct PairDown {
    int wk;             // K slices of a row tile
    int warps_r, warps_s;   // warps per routed / shared expert, each with wk / warps_* consecutive slices
    int upw_r, upw_s;   // units per slice
    int xcap;           // units of a warp's shared memory
    int warps_k;        // a K-quant shared expert's warps, behind the others
};
constexpr int kKqSteps = 4;   // row loads of a K-quant warp per item

// CTA-wide barrier that the K-quant warps reach in a loop of their own
__device__ __forceinline__ void cta_sync() { asm volatile("bar.sync 0;" ::: "memory"); }
// (a function of its own: its registers are not the products')
__device__ __noinline__ void pair_dispatch(const RouteParams& r, int* scratch, const int* ids) { build_dispatch(r, scratch, ids, 0); }

// grid = 1 + any number of CTAs (CTA 0: the dispatch step; items dealt round to the others).
// KQ: the last warps_k warps take a K-quant shared expert's rows of the tile: they form the token's intermediates (activation and Q8_1, a share
// of the blocks each), then a row (or two, of up to 16 sub-blocks) per step from weights asked for an item ahead.
template <int TYPE, bool KQ, int D, int THREADS, int CTAS>
__global__ void __launch_bounds__(THREADS, CTAS) pair_down_kernel(const __grid_constant__ RouteParams r, const __grid_constant__ GemvParams p,
                                                                  const __grid_constant__ PairExtras x, const __grid_constant__ PairDown c) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ int s_id[kPairItems * kMaxTopK];
    __shared__ float s_w[kPairItems * kMaxTopK];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    const int T = p.T, k = p.top_k;
    if (tid == 0) griddep_launch();   // (what follows in the stream waits for this grid before it touches the workspace)
    if (blockIdx.x == 0) {
        int* ids = reinterpret_cast<int*>(smem) + kDispatchSmemInts;
        for (int t = warp; t < T; t += nw) {
            const TopkSlot s = topk_select(r, r.router_logits + (size_t)t * r.E, lane, k);
            if (lane < k) ids[t * k + lane] = s.id;
        }
        __syncthreads();
        griddep_wait();
        if (tid < 256) pair_dispatch(r, reinterpret_cast<int*>(smem), ids);
        return;
    }
    const int cta = (int)blockIdx.x - 1, ctas = (int)gridDim.x - 1, n_items = T * (p.H >> 5), ni = (n_items - cta + ctas - 1) / ctas;
    // consecutive items share a row tile (the shared expert's then comes from L2)
    auto token = [&](int i) { const int n = cta + i * ctas; return n - n / T * T; };
    for (int i = warp; i < ni; i += nw) {
        const TopkSlot s = topk_select(r, r.router_logits + (size_t)token(i) * r.E, lane, k);
        if (lane < k) { s_id[i * kMaxTopK + lane] = s.id; s_w[i * kMaxTopK + lane] = s.w; }
    }
    __syncthreads();
    // this warp: slices s0 .. of expert slot `slot` (k = shared)
    const int nwr = k * c.warps_r;
    const bool routed = warp < nwr, idle = !routed && (p.nrows_shared == 0 || warp >= nwr + c.warps_s);
    const int slot = routed ? warp / c.warps_r : k, part = routed ? warp - slot * c.warps_r : warp - nwr;
    const int per = c.wk / (routed ? c.warps_r : max(c.warps_s, 1)), upw = routed ? c.upw_r : c.upw_s, gpw = upw >> 2;
    const int ncols = routed ? p.ncols_routed : p.ncols_shared, nb = idle ? 0 : ncols >> 5;
    const int u0 = min(nb, part * per * upw), nu_x = min(nb, u0 + per * upw) - u0, g0 = u0 >> 2, ng = (nu_x + 3) >> 2;
    const uint32_t xq = smem_u32(smem) + (uint32_t)(warp * c.xcap * 40), xd = xq + (uint32_t)c.xcap * 32;
    const int slices = k * c.wk + (KQ ? 1 : p.nrows_shared > 0 ? c.wk : 0);
    float* red = reinterpret_cast<float*>(smem + (size_t)nw * c.xcap * 40);   // [2][slice of every slot][32]
    if (KQ && !routed) {   // the K-quant warps' own loop (and that of warps with nothing to do)
        uint8_t* kx = smem + (size_t)nw * c.xcap * 40 + (size_t)2 * slices * 128;   // the token's intermediates, Q8_1
        const int kw = warp - nwr, ksub = x.F_s >> 5;
        const bool two = ksub <= 16, kq = kw < c.warps_k;
        const int ksb = two ? lane & 15 : lane, krow0 = kw * (32 / c.warps_k) + (two ? lane >> 4 : 0), kstep = two ? 2 : 1;
        SubBlock ks[kKqSteps];
        auto kq_load = [&](int i) {
            const size_t row = (size_t)((x.F_s >> 8) * kquant_block_bytes(x.type_down));
            const uint8_t* m = x.down + (size_t)((cta + i * ctas) / T * 32 + krow0) * row;
#pragma unroll
            for (int q = 0; q < kKqSteps; ++q)
                if (ksb < ksub) decode_sub(x.type_down, m + (size_t)(q * kstep) * row, ksb, ks[q]);
        };
        if (kq) kq_load(0);
        griddep_wait();
        for (int i = 0; i < ni; ++i) {
            float* mine = red + (i & 1) * (slices * 32);
            if (kq) {
                const int t = token(i);
                const float* u = x.rows + (size_t)t * x.F_s + lane;
                for (int b = kw; b < ksub; b += c.warps_k) {   // (act_q8_1_kernel's step)
                    const float uv = __ldcg(u + b * 32);
                    float v;
                    if (x.gate) v = silu_mul_ref(__ldcg(u + (size_t)T * x.F_s + b * 32), uv);
                    else { const float a = fmaxf(uv, 0.0f); v = a * a; }
                    float sum = v;
#pragma unroll
                    for (int q = 16; q > 0; q >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, q);
                    float d;
                    const int8_t qv = q8_1_warp(v, d);
                    uint8_t* blk = kx + b * kQ81Bytes;
                    reinterpret_cast<int8_t*>(blk)[4 + lane] = qv;
                    if (lane == 0) *reinterpret_cast<__half2*>(blk) = __halves2half2(__float2half(d), __float2half(sum));
                }
                asm volatile("bar.sync 3, %0;" ::"r"(c.warps_k * 32) : "memory");
#pragma unroll
                for (int q = 0; q < kKqSteps; ++q) {
                    float v = ksb < ksub ? add_dot(x.type_down, 0.0f, ks[q], kx + ksb * kQ81Bytes) : 0.0f;
                    if (!two) v += __shfl_xor_sync(0xffffffffu, v, 16);
#pragma unroll
                    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                    if (two ? (lane & 15) == 0 : lane == 0) mine[k * c.wk * 32 + krow0 + q * kstep] = v;
                }
                if (i + 1 < ni) kq_load(i + 1);
            }
            cta_sync();
        }
        return;
    }
    const int64_t tb = Tiled<TYPE>::tile_bytes(ncols);
    auto tile_of = [&](int i) {
        const uint8_t* m = routed ? p.w_a + (size_t)s_id[i * kMaxTopK + slot] * p.stride_a : p.sh_a;
        return m + (size_t)((cta + i * ctas) / T) * tb;
    };
    auto row_of = [&](int i) { return routed ? token(i) * k + slot : T * k + token(i); };
    auto units = [&](int g) { return min(4, nu_x - 4 * g); };
    PairGroup<TYPE> ra[D], rb;
    const uint8_t* ta = idle ? nullptr : tile_of(0);
#pragma unroll
    for (int d = 0; d < D; ++d) fill_group<TYPE>(ra[d], ta, g0 + d, lane, d < ng ? units(d) : 0);
    griddep_wait();
    PairX xr;
    load_x(xr, p, row_of(0), u0, nu_x, lane);
    for (int i = 0; i < ni; ++i) {
        const bool more = i + 1 < ni;
        const uint8_t* na = idle ? nullptr : tile_of(more ? i + 1 : i);
        store_x<TYPE>(xq, xd, xr, nu_x, lane);
        if (more) load_x(xr, p, row_of(i + 1), u0, nu_x, lane);
        float* mine = red + (i & 1) * (slices * 32);
        float acc = 0.0f, none = 0.0f;
        int left = gpw, s = slot * c.wk + part * per;
        for (int gg = 0; gg < ng; gg += D) {
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const int g = gg + d;
                if (g < ng) {
                    const bool same = g + D < ng;
                    pair_group<TYPE, false, (D > 1)>(ra[d], rb, g0 + g, units(g), xq + (uint32_t)g * 128, xd + (uint32_t)g * 32, acc, none, same ? ta : na, nullptr,
                                            g0 + (same ? g + D : d), same ? units(g + D) : more ? units(d) : 0, lane);
                    if (--left == 0 || g + 1 == ng) { mine[s * 32 + lane] = acc; acc = 0.0f; left = gpw; ++s; }
                }
            }
        }
        if (!idle) for (const int end = slot * c.wk + (part + 1) * per; s < end; ++s) mine[s * 32 + lane] = 0.0f;   // (slices behind the row's end)
        cta_sync();   // (the other half of `red` is free again: its reader has come to this barrier too)
        if (warp == i % nwr) {
            const int n = cta + i * ctas, tile = n / T, t = n - tile * T, h = tile * 32 + lane;
            const float logit = KQ ? (x.logit ? __ldcg(x.logit + t) : 0.0f) : p.nrows_shared > 0 && p.sh_gate_logit ? __ldcg(p.sh_gate_logit + t) : 0.0f;
            auto slot_sum = [&](int j) {
                float v = mine[j * c.wk * 32 + lane];
                for (int q = 1; q < c.wk; ++q) v += mine[(j * c.wk + q) * 32 + lane];
                return v;
            };
            float sum = 0.0f;   // weighted_combine_kernel (chimere_kernels.cu:1551-1565): slots ascending
            for (int j = 0; j < k; ++j) {
                const float v = slot_sum(j);
                if (!KQ) p.pair_out[((size_t)t * k + j) * p.H + h] = v;   // (with KQ the rows between the launches lie there)
                sum = fmaf(s_w[i * kMaxTopK + j], v, sum);
            }
            if (KQ || p.nrows_shared > 0) {  // sigmoid_gate_add_kernel (scratch_pool.rs:266-277)
                const float v = KQ ? mine[k * c.wk * 32 + lane] : slot_sum(k);
                if (!KQ) p.pair_out[((size_t)T * k + t) * p.H + h] = v;
                sum = (KQ ? x.logit : p.sh_gate_logit) ? fmaf(v, sigmoid_ref(logit), sum) : v + sum;
            }
            p.y[(size_t)t * p.H + h] = sum;
            if (tile == 0 && lane < k) {
                r.topk_idx[t * k + lane] = s_id[i * kMaxTopK + lane];
                r.topk_w[t * k + lane] = s_w[i * kMaxTopK + lane];
            }
        }
        ta = na;
    }
}

// ------------------------------------------------------------------ launchers --------------
static bool pair_type(int t) { return t == CHIMERE_TYPE_Q4_0 || t == CHIMERE_TYPE_IQ3_S; }

static bool pair_down_geom(const GemvParams& d, const PairExtras& x, PairDown& c, int& warps) {
    const bool sh = d.nrows_shared > 0;
    c.wk = tiled_down_geom(d.type_routed, d.ncols_routed, d.type_shared, sh ? d.ncols_shared : 0, d.T).wk;
    c.upw_r = tiled_slice_units(d.type_routed, d.ncols_routed, c.wk);
    c.upw_s = sh ? tiled_slice_units(d.type_shared, d.ncols_shared, c.wk) : 0;
    // as many warps per routed expert as 16 warps allow beside the shared expert's, which has one per slice
    c.warps_s = sh ? c.wk : 0;
    c.warps_k = !x.type ? 0 : x.F_s <= 512 ? 4 : 8;   // (rows of up to 16 sub-blocks go two at a time)
    for (c.warps_r = c.wk; c.warps_r > 1 && d.top_k * c.warps_r + c.warps_s + c.warps_k > 16; c.warps_r >>= 1) {}
    warps = d.top_k * c.warps_r + c.warps_s + c.warps_k;
    const int xr = c.wk / c.warps_r * c.upw_r, xs = sh ? c.upw_s : 0;
    c.xcap = xr > xs ? xr : xs;
    return warps <= 16 && c.xcap <= 32;
}

// Whether a K-quant shared expert rides along (gate and up of one type, four-byte aligned super-blocks, rows that the kernels' lanes hold).
bool pairs_take_kquant(const chimere_moe_layer& w) {
    const bool dual = w.act == CHIMERE_ACT_SWIGLU;
    const uintptr_t words = (uintptr_t)w.sh_up | (uintptr_t)w.sh_gate, down = (uintptr_t)w.sh_down;
    auto aligned = [](int type, uintptr_t p) { return (p & (type == CHIMERE_TYPE_Q6_K ? 1 : 3)) == 0; };
    return dual && w.type_sh_gate == w.type_sh_up && w.H <= 1024 * kKqSub && w.F_s <= 1024 && aligned(w.type_sh_up, words) && aligned(w.type_sh_down, down);
}

bool pairs_run(const GemvParams& gu, const GemvParams& d, const PairExtras& x) {
    const bool sh = d.nrows_shared > 0;
    if (!pair_type(gu.type_routed) || !pair_type(d.type_routed) || (sh && (gu.type_shared != gu.type_routed || d.type_shared != d.type_routed))) return false;
    const uintptr_t ptrs = (uintptr_t)gu.w_a | (uintptr_t)gu.w_b | (uintptr_t)gu.sh_a | (uintptr_t)gu.sh_b | (uintptr_t)gu.stride_a | (uintptr_t)gu.stride_b |
                           (uintptr_t)gu.in_soa_q | (uintptr_t)gu.in_soa_q_stride | (uintptr_t)d.w_a | (uintptr_t)d.sh_a | (uintptr_t)d.stride_a |
                           (uintptr_t)d.in_soa_q | (uintptr_t)d.in_soa_q_stride;
    if (ptrs & 15) return false;
    const int wk = tiled_gate_up_geom(gu.type_routed, gu.type_shared, gu.H, sh).wk;
    if (gu.H % 128 || tiled_slice_units(gu.type_routed, gu.H, wk) > 32) return false;
    PairDown c;
    int warps;
    return pair_down_geom(d, x, c, warps);
}

// CTAs for n items: as many as are resident together, more only where a CTA's list would not hold its share
static int pair_grid(int n_items, int resident) {
    const int least = (n_items + kPairItems - 1) / kPairItems;
    const int g = n_items < resident ? n_items : resident;
    return g > least ? g : least;
}

template <int TYPE, bool DUAL, bool KQ, int D, int CTAS>
static cudaError_t launch_pair_gu(const RouteParams& r, const GemvParams& p, const PairExtras& x, int n_items, int wk, int upw, cudaStream_t stream) {
    const size_t smem = (size_t)wk * upw * 40 + (size_t)2 * (DUAL ? 2 : 1) * wk * 128;
    const int resident = CTAS * (8 / wk) * sm_count();
    int grid = pair_grid(n_items, resident);
    if (KQ) grid = grid > resident / CTAS ? grid : resident / CTAS;   // (a row per warp, where the pairs alone would not fill the SMs)
    return launch_pdl(pair_gate_up_kernel<TYPE, DUAL, KQ, D, CTAS>, dim3(grid), 32 * wk, smem, stream, r, p, x, upw);
}
template <int TYPE, bool KQ, int D, int THREADS, int CTAS>
static cudaError_t launch_pair_dn(const RouteParams& r, const GemvParams& p, const PairExtras& x, const PairDown& c, int threads, cudaStream_t stream) {
    const int nw = threads / 32, slices = p.top_k * c.wk + (KQ ? 1 : p.nrows_shared > 0 ? c.wk : 0);
    const size_t smem = (size_t)nw * c.xcap * 40 + (size_t)2 * slices * 128 + (KQ ? x.F_s / 32 * kQ81Bytes : 0), list = (size_t)(kDispatchSmemInts + p.T * p.top_k) * 4;
    return launch_pdl(pair_down_kernel<TYPE, KQ, D, THREADS, CTAS>, dim3(1 + pair_grid(p.T * (p.H / 32), CTAS * sm_count() - 1)), threads, smem > list ? smem : list, stream,
                      r, p, x, c);
}

template <int TYPE>
static cudaError_t launch_pair_gu_t(const RouteParams& r, const GemvParams& p, const PairExtras& x, int n_items, int wk, int upw, cudaStream_t stream) {
    // One group in flight per warp (and matrix), as many CTAs as then keep their registers: 24 tokens of 256 gated experts take 264 us in four layers
    // so, 279 with two groups (56 bytes spilled) and 289 with three CTAs of one (140 bytes); ungated ones 95 with three CTAs, 98 with two groups.
    if (p.act != CHIMERE_ACT_SWIGLU) return launch_pair_gu<TYPE, false, false, 1, 3>(r, p, x, n_items, wk, upw, stream);
    return x.type ? launch_pair_gu<TYPE, true, true, 1, 2>(r, p, x, n_items, wk, upw, stream) : launch_pair_gu<TYPE, true, false, 1, 2>(r, p, x, n_items, wk, upw, stream);
}
cudaError_t launch_pair_gate_up(const RouteParams& r, const GemvParams& p, const PairExtras& x, cudaStream_t stream) {
    const int wk = tiled_gate_up_geom(p.type_routed, p.type_shared, p.H, p.nrows_shared > 0).wk, upw = tiled_slice_units(p.type_routed, p.H, wk);
    const int n_items = p.T * ((p.nrows_shared >> 5) + p.top_k * (p.nrows_routed >> 5));
    return p.type_routed == CHIMERE_TYPE_IQ3_S ? launch_pair_gu_t<CHIMERE_TYPE_IQ3_S>(r, p, x, n_items, wk, upw, stream)
                                               : launch_pair_gu_t<CHIMERE_TYPE_Q4_0>(r, p, x, n_items, wk, upw, stream);
}

template <int TYPE>
static cudaError_t launch_pair_dn_t(const RouteParams& r, const GemvParams& p, const PairExtras& x, const PairDown& c, int threads, cudaStream_t stream) {
    if (x.type) return launch_pair_dn<TYPE, true, 3, 512, 1>(r, p, x, c, threads, stream);
    if (threads > 288) return launch_pair_dn<TYPE, false, 3, 512, 1>(r, p, x, c, threads, stream);
    // Up to one item per SM the whole tile is in flight at once.  Else two CTAs per SM with two groups in flight each, or three with one where
    // that saves a round of items (256 experts of 512 columns, H = 2048, us per layer: 5 tokens 26.8 / 23.1, 8: 30.9 / 31.9, 16: 49.6 / 47.7).
    const int n = p.T * (p.H / 32), sms = sm_count();
    if (n < sms) return launch_pair_dn<TYPE, false, 4, 288, 1>(r, p, x, c, threads, stream);
    if ((n + 2 * sms - 2) / (2 * sms - 1) <= (n + 3 * sms - 2) / (3 * sms - 1)) return launch_pair_dn<TYPE, false, 2, 288, 2>(r, p, x, c, threads, stream);
    return launch_pair_dn<TYPE, false, 1, 288, 3>(r, p, x, c, threads, stream);
}
cudaError_t launch_pair_down(const RouteParams& r, const GemvParams& p, const PairExtras& x, cudaStream_t stream) {
    PairDown c;
    int warps;
    if (!pair_down_geom(p, x, c, warps)) return cudaErrorInvalidValue;
    const int threads = 32 * (warps < 8 ? 8 : warps);   // (the dispatch step is written for 256)
    return p.type_routed == CHIMERE_TYPE_IQ3_S ? launch_pair_dn_t<CHIMERE_TYPE_IQ3_S>(r, p, x, c, threads, stream) : launch_pair_dn_t<CHIMERE_TYPE_Q4_0>(r, p, x, c, threads, stream);
}

}  // namespace chimere
