// router.cu -- routing front end of the MoE layer, one launch for T tokens:
//   router logits (+ shared-expert gate logit), softmax / sigmoid top-k, Q8_1 of the input rows,
//   dispatch permutation and the work list of the grouped GEMV kernels.
//
// Arithmetic order is the reference's, so that logits, probabilities, indices and weights are
// bit-identical to its kernels on the same GPU:
//   f32_gemv_kernel      chimere-server/kernels/chimere_kernels.cu:706-741
//   dot_product_kernel   chimere-server/src/scratch_pool.rs:243-261
//   topk_softmax         chimere-server/kernels/chimere_kernels.cu:1150-1223
//   ggml_quantize_q8_1   chimere-server/kernels/chimere_kernels.cu:1495-1523
#include "common.cuh"
#include "kernels.h"
#include "routing.cuh"

namespace chimere {

// Q8_1 of one 32-float block by one warp; lane = element.
__device__ __forceinline__ void quantize_block_q8_1(float xi, uint8_t* out, int lane, int8_t* plane_q, float* plane_d) {
    float sum = xi;
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
    float d;
    const int8_t q = q8_1_warp(xi, d);
    reinterpret_cast<int8_t*>(out)[4 + lane] = q;
    const __half dh = __float2half(d);
    if (lane == 0) *reinterpret_cast<__half2*>(out) = __halves2half2(dh, __float2half(sum));
    // the same block as planes (what the tiled GEMV kernels stream)
    plane_q[lane] = q;
    if (lane == 0) *plane_d = __half2float(dh);
}

// Q8_1 of a whole row by a CTA of 256, four elements per lane and four blocks per warp step: a third of the instructions of a block per
// warp (quantize_block_q8_1), same bits -- the sum's butterfly has its strides 16, 8 and 4 across lanes and 2 and 1 within one.
__device__ __forceinline__ void quantize_row_q8_1(const float* src, int H, uint8_t* out, int8_t* plane_q, float* plane_d, int tid, int lane, int warp) {
    const bool aligned = ((uintptr_t)src & 15) == 0;
    for (int f0 = warp * 32; f0 < H >> 2; f0 += 256) {
        const int f = f0 + lane;
        const bool on = f < H >> 2;
        float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (on) {
            if (aligned) { const float4 x = *reinterpret_cast<const float4*>(src + 4 * f); v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; }
            else
#pragma unroll
                for (int c = 0; c < 4; ++c) v[c] = src[4 * f + c];
        }
        float t[4];
        uint32_t m = 0u;   // largest magnitude: bit patterns of non-negative floats order like the values, with the NaNs above infinity
#pragma unroll
        for (int c = 0; c < 4; ++c) { t[c] = v[c]; m = max(m, __float_as_uint(fabsf(v[c]))); }
#pragma unroll
        for (int s = 4; s > 0; s >>= 1) {
            m = max(m, __shfl_xor_sync(0xffffffffu, m, s));
#pragma unroll
            for (int c = 0; c < 4; ++c) t[c] += __shfl_xor_sync(0xffffffffu, t[c], s);
        }
        const float sum = (t[0] + t[2]) + (t[1] + t[3]);
        float amax = __uint_as_float(m), d;
        int q[4];
        if (__all_sync(0xffffffffu, !on || (amax > 1e-25f && amax < 1e25f))) {
            d = div_by_recip(amax, 127.0f, 1.0f / 127.0f);
            const float r = __frcp_rn(d);
#pragma unroll
            for (int c = 0; c < 4; ++c) q[c] = round_int(div_by_recip(v[c], d, r));
        } else {   // (see q8_1_warp)
            amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
            for (int s = 4; s > 0; s >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, s));
            d = amax / 127.0f;
#pragma unroll
            for (int c = 0; c < 4; ++c) q[c] = amax == 0.0f ? 0 : (int)(int8_t)roundf(v[c] / d);
        }
        if (on) {
            const uint32_t w = (uint32_t)(q[0] & 255) | ((uint32_t)(q[1] & 255) << 8) | ((uint32_t)(q[2] & 255) << 16) | ((uint32_t)(q[3] & 255) << 24);
            uint8_t* blk = out + (size_t)(f >> 3) * kQ81Bytes;
            *reinterpret_cast<uint32_t*>(blk + 4 + 4 * (f & 7)) = w;
            *reinterpret_cast<uint32_t*>(plane_q + 4 * f) = w;
            if ((f & 7) == 0) {
                const __half dh = __float2half(d);
                *reinterpret_cast<__half2*>(blk) = __halves2half2(dh, __float2half(sum));
                plane_d[f >> 3] = __half2float(dh);
            }
        }
    }
}

// grid = (row tiles, token tiles), 256 threads; TOKENS_X: (token tiles, row tiles), for more than the 65535 token tiles that the
// second dimension holds.  Thread p owns partial sum p of every output of the tile: elements p, p+256, ... in ascending order, one
// fused multiply-add each.
template <int TT, int TE, bool TOKENS_X = false>
__global__ void __launch_bounds__(256) route_kernel(const RouteParams p) {
    extern __shared__ __align__(16) float smem_f[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int H = p.H, E = p.E;
    const int nrows = E + (p.shexp_gate_w ? 1 : 0);
    const int ttile = TOKENS_X ? blockIdx.x : blockIdx.y, rtile = TOKENS_X ? blockIdx.y : blockIdx.x;
    const int t0 = ttile * TT, r0 = rtile * TE;
    const int n_ttiles = TOKENS_X ? gridDim.x : gridDim.y, n_rtiles = TOKENS_X ? gridDim.y : gridDim.x;

    // ---- partial dot products; the router rows come from DRAM, so their loads go out first and the Q8_1 of
    //      this token tile's input rows (blocks dealt round-robin to the row tiles) runs while they are in flight ----
    float acc[TT][TE];
#pragma unroll
    for (int a = 0; a < TT; ++a)
#pragma unroll
        for (int b = 0; b < TE; ++b) acc[a][b] = 0.0f;
    const float* wrow[TE];
#pragma unroll
    for (int b = 0; b < TE; ++b) {
        const int r = r0 + b;
        wrow[b] = (r < E) ? p.router_w + (size_t)r * H : ((r == E && r < nrows) ? p.shexp_gate_w : nullptr);
    }
    constexpr int kStep = TE == 1 ? 12 : TE == 2 ? 8 : 2;   // elements per thread whose loads are in flight together
    for (int j0 = 0; j0 < H; j0 += kStep * 256) {
        float wv[kStep][TE];
#pragma unroll
        for (int i = 0; i < kStep; ++i) {
            const int j = j0 + i * 256 + tid;
#pragma unroll
            for (int b = 0; b < TE; ++b) wv[i][b] = (j < H && wrow[b]) ? __ldg(wrow[b] + j) : 0.0f;
        }
        if (j0 == 0) {
            // The router rows are constants of the layer: their loads were issued above, possibly while the previous
            // kernel of the stream was still running (programmatic launch).  Everything that kernel may have written
            // (the input rows) or may still be reading (the workspace) is touched only after this wait.
            griddep_wait();
            if (tid == 0) griddep_launch();   // the grouped GEMV that follows may bring its CTAs in; it waits for this grid itself
            const int nbH = H >> 5;
            const int nt = min(TT, p.T - t0);
            for (int q = rtile * 8 + warp; q < nt * nbH; q += n_rtiles * 8) {
                const int tt = q / nbH, b = q - tt * nbH;
                const float xi = p.x[(size_t)(t0 + tt) * H + b * 32 + lane];
                quantize_block_q8_1(xi, p.x_q8 + ((size_t)(t0 + tt) * nbH + b) * kQ81Bytes, lane,
                                    p.x_soa_q + (size_t)(t0 + tt) * H + b * 32, p.x_soa_d + (size_t)(t0 + tt) * p.x_soa_d_stride + b);
            }
        }
        float xv[kStep][TT];
#pragma unroll
        for (int i = 0; i < kStep; ++i) {
            const int j = j0 + i * 256 + tid;
#pragma unroll
            for (int a = 0; a < TT; ++a) xv[i][a] = (j < H && t0 + a < p.T) ? p.x[(size_t)(t0 + a) * H + j] : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < kStep; ++i) {   // ascending j, one fused multiply-add each
            if (j0 + i * 256 + tid < H) {
#pragma unroll
                for (int a = 0; a < TT; ++a)
#pragma unroll
                    for (int b = 0; b < TE; ++b) acc[a][b] = fmaf(wv[i][b], xv[i][a], acc[a][b]);
            }
        }
    }
    float* red = smem_f;  // [TT*TE][256]
#pragma unroll
    for (int a = 0; a < TT; ++a)
#pragma unroll
        for (int b = 0; b < TE; ++b) red[(a * TE + b) * 256 + tid] = acc[a][b];
    __syncthreads();
    for (int o = warp; o < TT * TE; o += 8) {
        const float v = tree256(red + o * 256, lane);
        const int a = o / TE, b = o - a * TE;
        const int t = t0 + a, r = r0 + b;
        if (lane == 0 && t < p.T && r < nrows) {
            if (r < E) p.router_logits[(size_t)t * E + r] = p.router_bias ? v + p.router_bias[r] : v;
            else p.sh_gate_logit[t] = v;
        }
    }

    if (p.logits_only) return;

    // ---- last CTA of the token tile: scores and top-k ----
    __shared__ int s_flag;
    __shared__ int s_ids[TT * kMaxTopK];
    __syncthreads();   // every thread's writes are ordered before thread 0's counter increment, which releases them
    if (tid == 0) s_flag = (atom_add_acq_rel_gpu(&p.counters[kCtrRouteTile + ttile], 1) == n_rtiles - 1);   // ... and acquires the other CTAs'
    __syncthreads();
    if (!s_flag) return;
    if (tid == 0) p.counters[kCtrRouteTile + ttile] = 0;
    for (int a = warp; a < TT; a += 8) {
        const int t = t0 + a;
        if (t < p.T) topk_warp(p, p.router_logits + (size_t)t * E, t, lane, s_ids + a * p.top_k);
    }

    // ---- last token tile overall: dispatch permutation and work list ----
    if (n_ttiles == 1) {
        // the only token tile: its ids are all in shared memory
        __syncthreads();
        build_dispatch(p, reinterpret_cast<int*>(smem_f), s_ids, 0);
        return;
    }
    __syncthreads();   // every thread's writes are ordered before thread 0's counter increment, which releases them
    if (tid == 0) s_flag = (atom_add_acq_rel_gpu(&p.counters[kCtrRouteAll], 1) == n_ttiles - 1);   // ... and acquires the other CTAs'
    __syncthreads();
    if (!s_flag) return;
    if (tid == 0) p.counters[kCtrRouteAll] = 0;
    build_dispatch(p, reinterpret_cast<int*>(smem_f), nullptr, (int)(TT * TE * 256) - kDispatchSmemInts);
}

// The same for the first step of a half-layer of a few tokens: x = rmsnorm(residual + hidden) * weight is formed here (in every CTA: a
// thread holds the very elements that it sums squares of and multiplies with its router rows) instead of by a launch in front
// that stands for 4 us of latency.  In add_residual_rmsnorm_kernel's order (gemv.cu).  The logits alone, and x's Q8_1 form; the
// residual is updated by the launch behind, when every CTA has read it.  H <= 256 * KS.
template <int TT, int KS>
__global__ void __launch_bounds__(256) route_norm_kernel(const RouteParams p, const float* hidden, const float* residual, const float* weight, float eps) {
    __shared__ float s_red[TT * 2][256];
    __shared__ float s_sq[TT][256];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, H = p.H, E = p.E, r0 = blockIdx.x * 2;
    const int nrows = E + (p.shexp_gate_w ? 1 : 0);
    float wv[KS][2], x[TT][KS], nw[KS];
#pragma unroll
    for (int b = 0; b < 2; ++b) {
        const int r = r0 + b;
        const float* row = r < E ? p.router_w + (size_t)r * H : r == E && r < nrows ? p.shexp_gate_w : nullptr;
#pragma unroll
        for (int i = 0; i < KS; ++i) wv[i][b] = row && i * 256 + tid < H ? __ldg(row + i * 256 + tid) : 0.0f;
    }
    griddep_wait();
    if (tid == 0) griddep_launch();
    float hv[TT][KS];
#pragma unroll
    for (int a = 0; a < TT; ++a)
#pragma unroll
        for (int i = 0; i < KS; ++i) {
            const bool on = a < p.T && i * 256 + tid < H;
            hv[a][i] = on ? hidden[(size_t)a * H + i * 256 + tid] : 0.0f;
            x[a][i] = on ? residual[(size_t)a * H + i * 256 + tid] : 0.0f;
        }
#pragma unroll
    for (int i = 0; i < KS; ++i) nw[i] = i * 256 + tid < H ? weight[i * 256 + tid] : 0.0f;
#pragma unroll
    for (int a = 0; a < TT; ++a) {
        float sq = 0.0f;
#pragma unroll
        for (int i = 0; i < KS; ++i) {
            x[a][i] = hv[a][i] + x[a][i];
            if (i * 256 + tid < H) sq = fmaf(x[a][i], x[a][i], sq);
        }
        s_sq[a][tid] = sq;
    }
    __syncthreads();
    float acc[TT][2];
#pragma unroll
    for (int a = 0; a < TT; ++a) {
        const float total = __shfl_sync(0xffffffffu, tree256(s_sq[a], lane), 0);
        const float rms = sqrtf(total / (float)H + eps);
        const float inv_rms = 1.0f / rms;
        acc[a][0] = acc[a][1] = 0.0f;
#pragma unroll
        for (int i = 0; i < KS; ++i) {
            x[a][i] = x[a][i] * inv_rms * nw[i];
            if (i * 256 + tid < H) { acc[a][0] = fmaf(wv[i][0], x[a][i], acc[a][0]); acc[a][1] = fmaf(wv[i][1], x[a][i], acc[a][1]); }
        }
        s_red[2 * a][tid] = acc[a][0];
        s_red[2 * a + 1][tid] = acc[a][1];
    }
    // Q8_1: elements i * 256 + 32 * warp .. of a token are block 8 * i + warp, lane = element; (token, i) pairs are dealt to the CTAs
    for (int q = blockIdx.x; q < p.T * KS; q += gridDim.x) {
        const int t = q / KS, b = (q - t * KS) * 8 + warp;
        float xi = 0.0f;
#pragma unroll
        for (int a = 0; a < TT; ++a)
#pragma unroll
            for (int i = 0; i < KS; ++i)
                if (q == a * KS + i) xi = x[a][i];
        if (b < H >> 5) quantize_block_q8_1(xi, p.x_q8 + ((size_t)t * (H >> 5) + b) * kQ81Bytes, lane, p.x_soa_q + (size_t)t * H + b * 32, p.x_soa_d + (size_t)t * p.x_soa_d_stride + b);
    }
    __syncthreads();
    for (int o = warp; o < TT * 2; o += 8) {
        const float v = tree256(s_red[o], lane);
        const int t = o >> 1, r = r0 + (o & 1);
        if (lane == 0 && t < p.T && r < nrows) {
            if (r < E) p.router_logits[(size_t)t * E + r] = p.router_bias ? v + p.router_bias[r] : v;
            else p.sh_gate_logit[t] = v;
        }
    }
}

// Larger batches, as a register-tiled product.  The order of the additions is fixed (256 partial sums per output, partial p over
// elements p, p+256, ..., then a tree of strides 128 .. 1), but a single thread can follow it: taking the partials in
// bit-reversed order turns the tree into one over neighbours, which a binary counter of pending sums walks with one add per
// partial.  So a thread owns 4 x 4 outputs (tokens x experts) and nothing is exchanged until the top levels of the tree, which
// are split over WP warps of the CTA and meet in shared memory once at the end.
//   route_prep_kernel : one CTA per token or router row: the row rewritten in that order (below), and for a token the Q8_1 form
//                       and the shared expert's gate logit
//   route_tile_kernel : CTA tile of 32 tokens x 16 experts (16 x 16 in small batches), its eight warps with an eighth of the partials each; chunks of two
//                       partials come through a ring of bulk copies of every warp's own (no CTA barrier until the end)
//   route_topk_kernel : scores and top-k, one warp per token; the last CTA does the dispatch
// Bound by the FMA pipe and its operands: 8 LDS.128 per 64 multiply-adds and thread.  (The form before it kept one partial of 32
// outputs per thread and passed all 256 partials of every output through shared memory: 563 us at T = 8192, E = 256, H = 2048, 68 us
// at T = 512.  Tiles of 64 x 32 with the partials split over two warps read half the bytes per output, but a CTA of them takes 40 us
// whatever the batch, and at T = 8192 they are no faster.)
// Order of a row's copy: [chunk of 2 partials][row][2 partials x NQ x 4 elements, 4 floats of padding]; partial number n stands for
// p = bit-reversed n.  The padding puts the rows a warp reads together on different banks.
constexpr int kRoutePartials = 2, kRouteChunks = 256 / kRoutePartials;
__host__ __device__ constexpr int route_pitch(int nq) { return 4 * kRoutePartials * nq + 4; }   // floats of a row in a chunk
__host__ __device__ constexpr int route_nq(int H) { return (H + 1023) / 1024; }
static size_t route_scratch_floats(int T, int E, int H) { return (size_t)(T + E) * kRouteChunks * route_pitch(route_nq(H)); }

template <int NQ>
__global__ void __launch_bounds__(256) route_prep_kernel(const RouteParams p) {
    __shared__ float red[256];
    constexpr int kPitch = route_pitch(NQ);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, H = p.H;
    const bool token = (int)blockIdx.x < p.T;
    const int row = token ? blockIdx.x : blockIdx.x - p.T, rows = token ? p.T : p.E;
    const float* src = token ? p.x + (size_t)row * H : p.router_w + (size_t)row * H;
    float v[4 * NQ];
    griddep_wait();
    if (tid == 0) griddep_launch();
#pragma unroll
    for (int i = 0; i < 4 * NQ; ++i) v[i] = i * 256 + tid < H ? src[i * 256 + tid] : 0.0f;
    const int n = (int)(__brev((unsigned)tid) >> 24);
    float* dst = p.scratch + (token ? 0 : (size_t)p.T * kRouteChunks * kPitch);
    dst += ((size_t)(n / kRoutePartials) * rows + row) * kPitch + (n % kRoutePartials) * (4 * NQ);
#pragma unroll
    for (int q = 0; q < NQ; ++q) *reinterpret_cast<float4*>(dst + 4 * q) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    if (!token) return;
    if (p.shexp_gate_w) {
        float acc = 0.0f;
#pragma unroll
        for (int i = 0; i < 4 * NQ; ++i)
            if (i * 256 + tid < H) acc = fmaf(p.shexp_gate_w[i * 256 + tid], v[i], acc);
        red[tid] = acc;
    }
    quantize_row_q8_1(src, H, p.x_q8 + (size_t)row * (H >> 5) * kQ81Bytes, p.x_soa_q + (size_t)row * H, p.x_soa_d + (size_t)row * p.x_soa_d_stride, tid, lane, warp);
    if (p.shexp_gate_w) {
        __syncthreads();
        if (warp == 0) {
            const float g = tree256(red, lane);
            if (lane == 0) p.sh_gate_logit[row] = g;
        }
    }
}

// TA: tokens of a thread (tokens of a tile / 8)
template <int NQ, int TA> struct RouteTile {
    static constexpr int kTok = 8 * TA, kExp = 16, kOut = 4 * TA, kWarps = 8, kPitch = route_pitch(NQ), kSteps = kRouteChunks / kWarps;
    static constexpr int kStage = (kTok + kExp) * kPitch, kRing = TA == 2 && NQ > 2 ? 4 : 2;   // floats of a warp's stage; two CTAs per SM up to NQ = 2
    static constexpr int kLevels = 4, kPending = (kLevels - 1) * kOut * 256;   // pending sums of the levels above the first
    static constexpr size_t kSmem = ((size_t)kWarps * kRing * kStage + kPending) * 4;
    static_assert(kSteps == 1 << kLevels, "a warp's chunks are the leaves of its part of the tree");
    static_assert(kTok * kExp <= kRing * kStage, "the shares of the outputs meet in the ring's memory");
};

__device__ __forceinline__ float4 lds_f4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}

// grid = (expert tiles, token tiles)
template <int NQ, int TA>
__global__ void __launch_bounds__(256, 2) route_tile_kernel(const RouteParams p) {
    using R = RouteTile<NQ, TA>;
    extern __shared__ __align__(128) float smem_f[];
    __shared__ __align__(8) uint64_t s_full[R::kWarps][R::kRing];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int T = p.T, E = p.E, t0 = blockIdx.y * R::kTok, e0 = blockIdx.x * R::kExp;
    float* ring = smem_f + warp * (R::kRing * R::kStage);
    uint64_t* full = s_full[warp];
    const uint32_t xb = (uint32_t)min(R::kTok, T - t0) * (R::kPitch * 4), wb = (uint32_t)min(R::kExp, E - e0) * (R::kPitch * 4);
    const float* xsrc = p.scratch + ((size_t)(warp * R::kSteps) * T + t0) * R::kPitch;
    const float* wsrc = p.scratch + ((size_t)T * kRouteChunks + (size_t)(warp * R::kSteps) * E + e0) * R::kPitch;
    auto ask = [&](int slot) {   // the warp's next chunk (lane 0)
        mbar_expect_tx(&full[slot], xb + wb);
        bulk_g2s(ring + slot * R::kStage, xsrc, xb, &full[slot]);
        bulk_g2s(ring + slot * R::kStage + R::kTok * R::kPitch, wsrc, wb, &full[slot]);
        xsrc += (size_t)T * R::kPitch;
        wsrc += (size_t)E * R::kPitch;
    };
    if (lane == 0) {
        for (int i = 0; i < R::kRing; ++i) mbar_init(&full[i], 1);
        mbar_fence_init();
    }
    griddep_wait();
    if (tid == 0) griddep_launch();
    if (lane == 0)
        for (int k = 0; k < R::kRing; ++k) ask(k);
    __syncwarp();
    // this thread: tokens tg + 8 a, experts eg + 4 b
    const int tg = lane & 7, eg = lane >> 3;
    const uint32_t xs0 = smem_u32(ring) + 4u * (tg * R::kPitch), ws0 = smem_u32(ring) + 4u * ((R::kTok + eg) * R::kPitch);
    // pending sums: the first level's in registers, the others in shared memory, thread beside thread (a register file of them
    // would leave one CTA per SM, local memory costs a small batch 10 us of first touches)
    float* st = smem_f + R::kWarps * R::kRing * R::kStage + tid;
    float pend[R::kOut], v[R::kOut];
    bool ok = true;
    uint32_t phase = 0;
    int slot = 0;
    for (int k = 0; k < R::kSteps; ++k) {
        if (!mbar_wait(&full[slot], phase)) { ok = false; break; }
        const uint32_t xs = xs0 + 4u * (slot * R::kStage), ws = ws0 + 4u * (slot * R::kStage);
#pragma unroll
        for (int j = 0; j < kRoutePartials; ++j) {
            float acc[R::kOut];
#pragma unroll
            for (int i = 0; i < R::kOut; ++i) acc[i] = 0.0f;
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                float4 w[4];
#pragma unroll
                for (int b = 0; b < 4; ++b) w[b] = lds_f4(ws + 4u * (4 * b * R::kPitch + (j * NQ + q) * 4));
#pragma unroll
                for (int a = 0; a < TA; ++a) {
                    const float4 x = lds_f4(xs + 4u * (8 * a * R::kPitch + (j * NQ + q) * 4));
#pragma unroll
                    for (int b = 0; b < 4; ++b) acc[4 * a + b] = fmaf(w[b].x, x.x, acc[4 * a + b]);   // ascending elements, one fused multiply-add each
#pragma unroll
                    for (int b = 0; b < 4; ++b) acc[4 * a + b] = fmaf(w[b].y, x.y, acc[4 * a + b]);
#pragma unroll
                    for (int b = 0; b < 4; ++b) acc[4 * a + b] = fmaf(w[b].z, x.z, acc[4 * a + b]);
#pragma unroll
                    for (int b = 0; b < 4; ++b) acc[4 * a + b] = fmaf(w[b].w, x.w, acc[4 * a + b]);
                }
            }
#pragma unroll
            for (int i = 0; i < R::kOut; ++i) v[i] = j == 0 ? acc[i] : v[i] + acc[i];
        }
        __syncwarp();   // every lane has read the slot
        if (lane == 0 && k + R::kRing < R::kSteps) ask(slot);
        if (++slot == R::kRing) { slot = 0; phase ^= 1u; }
        // the binary counter: v completes level after level as long as that level has a pending left half
        if (!(k & 1)) {
#pragma unroll
            for (int i = 0; i < R::kOut; ++i) pend[i] = v[i];
            continue;
        }
#pragma unroll
        for (int i = 0; i < R::kOut; ++i) v[i] += pend[i];
#pragma unroll
        for (int l = 1; l < R::kLevels; ++l) {
            float* sl = st + (l - 1) * R::kOut * 256;
            if ((k >> l) & 1) {
#pragma unroll
                for (int i = 0; i < R::kOut; ++i) v[i] += sl[i * 256];
            } else {
#pragma unroll
                for (int i = 0; i < R::kOut; ++i) sl[i * 256] = v[i];
                break;
            }
        }
    }
    if (!ok && lane == 0) {
        if (p.status) atomicOr(p.status, kStatusWaitTimeout);
        for (int i = 0; i < R::kRing; ++i) { mbar_wait(&full[i], 0); mbar_wait(&full[i], 1); }   // its copies have to land before this memory goes away
    }
    __syncwarp();
    // the warps' shares of every output, each in its own ring's memory (row pitch 17: the lanes of a store on different banks)
#pragma unroll
    for (int a = 0; a < TA; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) ring[(tg + 8 * a) * 17 + eg + 4 * b] = v[4 * a + b];
    __syncthreads();
    for (int o = tid; o < R::kTok * R::kExp; o += 256) {
        const int r = o / R::kExp, c = o % R::kExp, t = t0 + r, e = e0 + c;
        float s[R::kWarps];
#pragma unroll
        for (int g = 0; g < R::kWarps; ++g) s[g] = smem_f[g * (R::kRing * R::kStage) + r * 17 + c];
        const float sum = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
        if (t < T && e < E) p.router_logits[(size_t)t * E + e] = p.router_bias ? sum + p.router_bias[e] : sum;
    }
}

// Scores and top-k, one warp per token; unless the dispatch follows as launches of its own (hist: its counts, a chunk of `tokens` per CTA), the
// last CTA does it (tokens = 0: nobody here).
constexpr int kTopkIdsRoom = 4096;
__global__ void __launch_bounds__(256) route_topk_kernel(const RouteParams p, int32_t* hist, int tokens) {
    extern __shared__ __align__(16) float smem_f[];
    __shared__ int s_flag;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    griddep_wait();
    if (tid == 0) griddep_launch();
    if (hist) {
        int* cnt = reinterpret_cast<int*>(smem_f);
        int* ids = cnt + 256;
        cnt[tid] = 0;
        const int t0 = blockIdx.x * tokens, n = min(tokens, p.T - t0);
        for (int a = warp; a < n; a += 8) topk_warp(p, p.router_logits + (size_t)(t0 + a) * p.E, t0 + a, lane, ids + a * p.top_k);
        __syncthreads();
        if (tid < n * p.top_k) atomicAdd(cnt + ids[tid], 1);
        __syncthreads();
        hist[(size_t)blockIdx.x * 256 + tid] = cnt[tid];
        return;
    }
    const int t = blockIdx.x * 8 + warp;
    if (t < p.T) topk_warp(p, p.router_logits + (size_t)t * p.E, t, lane, nullptr);
    if (tokens == 0) return;
    __syncthreads();   // every thread's writes are ordered before thread 0's counter increment, which releases them
    if (tid == 0) s_flag = (atom_add_acq_rel_gpu(&p.counters[kCtrRouteAll], 1) == (int)gridDim.x - 1);   // ... and acquires the other CTAs'
    __syncthreads();
    if (!s_flag) return;
    if (tid == 0) p.counters[kCtrRouteAll] = 0;
    build_dispatch(p, reinterpret_cast<int*>(smem_f), nullptr, kTopkIdsRoom);
}

// ---- dispatch of a large batch in three small launches --------------------------------------
// One CTA sorting tens of thousands of pairs is a serial tail of hundreds of microseconds, so large batches split
// the same stable counting sort over the GPU: chunks of up to 128 consecutive pairs are counted per expert -- by the top-k
// kernel, where a chunk is few tokens, else by a launch --, a warp per expert turns the counts into every chunk's first position within
// it and the last CTA the totals into offsets (scan), and the chunks place their own pairs (place); whoever finishes last writes the GEMV
// work list.  Scratch: hist[chunks][256] + 260 ints behind it, zero before and after (it shares memory with the combine
// counters of the down stage, which need zeros).

__global__ void __launch_bounds__(kDispatchChunk) dispatch_hist_kernel(const RouteParams p, int32_t* hist, int chunk) {
    __shared__ int s_ids[kDispatchChunk];
    const int tid = threadIdx.x, P = p.T * p.top_k, q = blockIdx.x * chunk + tid;
    const int istr = p.idx_stride > 1 ? p.idx_stride : 1;
    griddep_wait();
    if (tid == 0) griddep_launch();
    int e = tid < chunk && q < P ? __ldcg(p.topk_idx + (size_t)q * istr) : -1;
    s_ids[tid] = (e >= 0 && e < p.E) ? e : -1;
    __syncthreads();
    for (int x = tid; x < 256; x += kDispatchChunk) {
        int c = 0;
#pragma unroll 8
        for (int i = 0; i < kDispatchChunk; ++i) c += (s_ids[i] == x);
        hist[(size_t)blockIdx.x * 256 + x] = c;
    }
}

// The last step of both scans, by 256 threads, thread = expert: pair counts to offsets and to the first work entries.
__device__ __forceinline__ void scan_totals(const RouteParams& p, int32_t* ent_base, int cnt, int* scan) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nent = (cnt + kMaxGroupTokens - 1) / kMaxGroupTokens;
    int incl_c = cnt, incl_n = nent;
#pragma unroll
    for (int sft = 1; sft < 32; sft <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, incl_c, sft), b = __shfl_up_sync(0xffffffffu, incl_n, sft);
        if (lane >= sft) { incl_c += a; incl_n += b; }
    }
    if (lane == 31) { scan[warp] = incl_c; scan[8 + warp] = incl_n; }
    dispatch_sync();
    int base_c = 0, base_n = 0;
    for (int w = 0; w < warp; ++w) { base_c += scan[w]; base_n += scan[8 + w]; }
    if (tid < p.E) p.offsets[tid] = base_c + incl_c - cnt;
    ent_base[tid] = base_n + incl_n - nent;
    if (tid == 255) { p.offsets[p.E] = base_c + incl_c; ent_base[256] = base_n + incl_n; }
}

// hist[chunk][e] becomes the number of pairs of expert e in earlier chunks.  Many chunks: a warp per expert, a run of consecutive chunks per
// lane, the CTA that finishes last does the totals (512 chunks, the launch alone: 13.6 us, where one CTA for all experts takes 22.5, of one SM's loads).
constexpr int kScanBatch = 16;
__global__ void __launch_bounds__(256) dispatch_scan_kernel(const RouteParams p, int32_t* hist, int nchunks) {
    __shared__ int scan[16];
    __shared__ int s_flag;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, e = blockIdx.x * 8 + warp;
    griddep_wait();
    if (tid == 0) griddep_launch();
    int32_t* ent_base = hist + (size_t)nchunks * 256;   // [257] first routed entry of each expert, then their number; [259] CTAs done here
    {
        const int per = (nchunks + 31) / 32, c0 = min(nchunks, lane * per), c1 = min(nchunks, c0 + per);
        int32_t* col = hist + e;
        int sum = 0;
        for (int c = c0; c < c1; c += kScanBatch) {
            int v[kScanBatch];
#pragma unroll
            for (int i = 0; i < kScanBatch; ++i) v[i] = c + i < c1 ? __ldcg(col + (size_t)(c + i) * 256) : 0;
#pragma unroll
            for (int i = 0; i < kScanBatch; ++i) sum += v[i];
        }
        int run = sum;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, run, s);
            if (lane >= s) run += a;
        }
        if (lane == 31) ent_base[e] = run;   // (the expert's pairs, until the last CTA has them)
        run -= sum;
        for (int c = c0; c < c1; c += kScanBatch) {
            int v[kScanBatch];
#pragma unroll
            for (int i = 0; i < kScanBatch; ++i) v[i] = c + i < c1 ? __ldcg(col + (size_t)(c + i) * 256) : 0;
#pragma unroll
            for (int i = 0; i < kScanBatch; ++i)
                if (c + i < c1) { col[(size_t)(c + i) * 256] = run; run += v[i]; }
        }
    }
    __syncthreads();   // every thread's writes are ordered before thread 0's counter increment, which releases them
    if (tid == 0) s_flag = (atom_add_acq_rel_gpu(ent_base + 259, 1) == (int)gridDim.x - 1);   // ... and acquires the other CTAs'
    __syncthreads();
    if (!s_flag) return;
    if (tid == 0) ent_base[259] = 0;
    scan_totals(p, ent_base, tid < p.E ? __ldcg(ent_base + tid) : 0, scan);
}
// Few chunks: one CTA, thread = (quarter of the chunks, expert), a quarter of up to 16 chunks in registers between the two passes; no counter and
// no second look at the totals (32 chunks, the launch alone: 9.0 -> 4.2).  Route entry, us, 32 CTAs / one: 256 experts of H = 2048, 512 tokens (32 chunks) 59.4 / 55.0, 1024 (64) 93.0 / 88.2; 200 of
// H = 1152, 1024: 92.6 / 87.2 (88.9 when this was a launch behind one that counted).
constexpr int kScanFewChunks = 4 * kScanBatch;
__global__ void __launch_bounds__(1024) dispatch_scan_few_kernel(const RouteParams p, int32_t* hist, int nchunks) {
    __shared__ int scan[16];
    __shared__ int part[4][256];
    const int e = threadIdx.x & 255, quarter = threadIdx.x >> 8, per = (nchunks + 3) / 4, c0 = quarter * per;
    int32_t* col = hist + (size_t)c0 * 256 + e;
    griddep_wait();
    if (threadIdx.x == 0) griddep_launch();
    int v[kScanBatch], sum = 0;
#pragma unroll
    for (int i = 0; i < kScanBatch; ++i) v[i] = i < per && c0 + i < nchunks ? __ldcg(col + (size_t)i * 256) : 0;
#pragma unroll
    for (int i = 0; i < kScanBatch; ++i) sum += v[i];
    part[quarter][e] = sum;
    __syncthreads();
    int run = 0;
    for (int q = 0; q < quarter; ++q) run += part[q][e];
#pragma unroll
    for (int i = 0; i < kScanBatch; ++i)
        if (i < per && c0 + i < nchunks) { col[(size_t)i * 256] = run; run += v[i]; }
    if (quarter > 0) return;
    scan_totals(p, hist + (size_t)nchunks * 256, e < p.E ? part[0][e] + part[1][e] + part[2][e] + part[3][e] : 0, scan);
}

__global__ void __launch_bounds__(kDispatchChunk) dispatch_place_kernel(const RouteParams p, int32_t* hist, int nchunks, int chunk) {
    __shared__ int s_ids[kDispatchChunk];
    __shared__ int s_last;
    const int tid = threadIdx.x, P = p.T * p.top_k, q = blockIdx.x * chunk + tid;
    const int istr = p.idx_stride > 1 ? p.idx_stride : 1;
    griddep_wait();
    if (tid == 0) griddep_launch();
    int e = tid < chunk && q < P ? __ldcg(p.topk_idx + (size_t)q * istr) : -1;
    if (e < 0 || e >= p.E) e = -1;
    s_ids[tid] = e;
    __syncthreads();
    if (e >= 0) {
        int rank = 0;
        for (int i = 0; i < tid; ++i) rank += (s_ids[i] == e);
        p.perm[__ldcg(p.offsets + e) + __ldcg(hist + (size_t)blockIdx.x * 256 + e) + rank] = q;
    }
    __syncthreads();
    for (int x = tid; x < 256; x += kDispatchChunk) hist[(size_t)blockIdx.x * 256 + x] = 0;   // back to zero for whoever shares this memory
    // ---- the chunk that finishes last writes the work list ----
    int32_t* ent_base = hist + (size_t)nchunks * 256;
    int32_t* done = ent_base + 258;
    __syncthreads();   // every thread's writes are ordered before thread 0's counter increment, which releases them
    if (tid == 0) s_last = (atom_add_acq_rel_gpu(done, 1) == nchunks - 1);   // ... and acquires the other CTAs'
    __syncthreads();
    if (!s_last) return;
    __shared__ int s_ent[257], s_off[257];
    for (int x = tid; x < 257; x += kDispatchChunk) { s_ent[x] = __ldcg(ent_base + x); s_off[x] = x <= p.E ? __ldcg(p.offsets + x) : 0; }
    __syncthreads();
    const int sgt = shared_group_tokens(p.T);
    const int nsh = (p.has_shared && p.list_mode != 2) ? (p.T + sgt - 1) / sgt : 0;
    int total_routed = p.list_mode == 0 ? s_ent[256] : 0;
    if (nsh + total_routed > p.list_capacity) {
        total_routed = max(0, p.list_capacity - nsh);
        if (tid == 0 && p.status) atomicOr(p.status, kStatusListFull);
    }
    for (int i = tid; i < nsh; i += kDispatchChunk) {
        int* ent = p.group_list + kListHeader + kListEntry * i;
        const int t0 = i * sgt, mm = min(sgt, p.T - t0);
        ent[0] = -1; ent[1] = t0; ent[2] = mm; ent[3] = 0;
        for (int j = 0; j < kMaxGroupTokens; ++j) ent[4 + j] = j < mm ? p.T * p.top_k + t0 + j : 0;
    }
    for (int idx = tid; idx < total_routed; idx += kDispatchChunk) {
        int lo = 0, hi = 256;   // ent_base[lo] <= idx < ent_base[hi]
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_ent[mid] <= idx) lo = mid; else hi = mid;
        }
        const int ex = lo, i = idx - s_ent[ex], o = s_off[ex], cnt = s_off[ex + 1] - o;
        const int mm = min(kMaxGroupTokens, cnt - i * kMaxGroupTokens);
        int* ent = p.group_list + kListHeader + kListEntry * (nsh + idx);
        ent[0] = ex; ent[1] = o + i * kMaxGroupTokens; ent[2] = mm; ent[3] = 0;
        for (int j = 0; j < kMaxGroupTokens; ++j) ent[4 + j] = j < mm ? __ldcg(p.perm + o + i * kMaxGroupTokens + j) : 0;
    }
    __syncthreads();
    if (tid == 0) {
        p.group_list[0] = total_routed + nsh; p.group_list[1] = total_routed; p.group_list[2] = nsh; p.group_list[3] = 0;
        *done = 0;
    }
    for (int x = tid; x < 258; x += kDispatchChunk) ent_base[x] = 0;
}

// counted: the top-k kernel has left the counts
static cudaError_t launch_dispatch_split(const RouteParams& p, bool counted, cudaStream_t stream) {
    const int nchunks = dispatch_chunks(p.T, p.top_k), chunk = dispatch_tokens(p.top_k) * p.top_k;
    cudaError_t e = cudaSuccess;
    if (!counted) e = launch_pdl(dispatch_hist_kernel, dim3(nchunks), kDispatchChunk, 0, stream, p, p.dispatch_scratch, chunk);
    if (e == cudaSuccess)
        e = nchunks <= kScanFewChunks ? launch_pdl(dispatch_scan_few_kernel, dim3(1), 1024, 0, stream, p, p.dispatch_scratch, nchunks)
                                      : launch_pdl(dispatch_scan_kernel, dim3(32), 256, 0, stream, p, p.dispatch_scratch, nchunks);
    if (e == cudaSuccess) e = launch_pdl(dispatch_place_kernel, dim3(nchunks), kDispatchChunk, 0, stream, p, p.dispatch_scratch, nchunks, chunk);
    return e;
}
// Batches from this many pairs on take the three-launch dispatch (below, the single CTA at the router's end is faster).
constexpr int kSplitDispatchPairs = 4096;
static bool use_split_dispatch(const RouteParams& p) { return p.dispatch_scratch != nullptr && p.T * p.top_k >= kSplitDispatchPairs; }

// ---- counters of the expert-parallel exchange by peer stores (see the kernels further down) ----
__device__ __forceinline__ int ld_acquire_sys(const int32_t* p) { int v; asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory"); return v; }
__device__ __forceinline__ void red_release_sys_add(int32_t* p, int v) { asm volatile("red.release.sys.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
// true when *flag reached `expect` within the bound
__device__ __forceinline__ bool wait_flag(const int32_t* flag, int expect) {
    for (int it = 0; it < (1 << 22); ++it) {
        if (ld_acquire_sys(flag) >= expect) return true;
        __nanosleep(40);
    }
    return false;
}

// The dispatch step alone, for callers that bring their own expert ids in p.topk_idx.  An expert-parallel owner rank
// whose rows arrive by peer stores first waits (bounded) for the source ranks' counters and takes them down.
constexpr int kPermuteIdsRoom = 8192;
__global__ void __launch_bounds__(256) permute_kernel(const RouteParams p) {
    extern __shared__ __align__(16) float smem_f[];
    if (p.wait_flags) {
        if ((int)threadIdx.x < p.wait_n) {
            if (!wait_flag(p.wait_flags + threadIdx.x, p.wait_expect) && p.status) atomicOr(p.status, kStatusWaitTimeout);
            p.wait_flags[threadIdx.x] = 0;
        }
        __syncthreads();
    }
    build_dispatch(p, reinterpret_cast<int*>(smem_f), nullptr, kPermuteIdsRoom);
}

// Final step of an expert-parallel layer on the tokens' home rank: routing-weighted sum of the k expert
// rows of every token in slot order (weighted_combine_kernel, chimere_kernels.cu:1551-1565) plus the
// sigmoid-gated shared expert (sigmoid_gate_add_kernel, scratch_pool.rs:266-277).
// HBM-bound: T * (k + 1) rows in, T out.  Four elements per thread and every row's load issued before the first is used
// (k <= kMaxTopK): 161 us with one element and one load at a time at T = 8192, k = 8, H = 2048.  ALIGNED: rows, shared rows and y
// lie on 16-byte boundaries and go as one access of four elements; a caller's y or rows may lie on any float.
template <bool ALIGNED>
__device__ __forceinline__ float4 ld_row4(const float* p) {
    if (ALIGNED) return __ldcs(reinterpret_cast<const float4*>(p));
    return make_float4(__ldcs(p), __ldcs(p + 1), __ldcs(p + 2), __ldcs(p + 3));
}
template <bool ALIGNED>
__global__ void __launch_bounds__(256) ep_finish_kernel(const float* rows, const int32_t* slot, const float* topk_w, const float* shared_rows, const float* sh_logit,
                                                        float* y, int T, int H, int k) {
    griddep_wait();
    if (threadIdx.x == 0) griddep_launch();
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int h4 = H >> 2;
    if (idx >= (int64_t)T * h4) return;
    const int t = (int)(idx / h4), h = (int)(idx - (int64_t)t * h4) * 4;
    float4 v[kMaxTopK], sh;
    float w[kMaxTopK];
#pragma unroll
    for (int j = 0; j < kMaxTopK; ++j)
        if (j < k) {
            const size_t r = slot ? (size_t)slot[t * k + j] : (size_t)t * k + j;   // where pair (t, j) came back
            v[j] = ld_row4<ALIGNED>(rows + r * H + h);
            w[j] = topk_w[(size_t)t * k + j];
        }
    if (shared_rows) sh = ld_row4<ALIGNED>(shared_rows + (size_t)t * H + h);
    float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int j = 0; j < kMaxTopK; ++j)
        if (j < k) { sum.x = fmaf(w[j], v[j].x, sum.x); sum.y = fmaf(w[j], v[j].y, sum.y); sum.z = fmaf(w[j], v[j].z, sum.z); sum.w = fmaf(w[j], v[j].w, sum.w); }
    if (shared_rows) {
        if (sh_logit) {
            const float g = sigmoid_ref(sh_logit[t]);
            sum.x = fmaf(sh.x, g, sum.x); sum.y = fmaf(sh.y, g, sum.y); sum.z = fmaf(sh.z, g, sum.z); sum.w = fmaf(sh.w, g, sum.w);
        } else { sum.x += sh.x; sum.y += sh.y; sum.z += sh.z; sum.w += sh.w; }
    }
    float* out = y + (size_t)t * H + h;
    if (ALIGNED) *reinterpret_cast<float4*>(out) = sum;
    else { out[0] = sum.x; out[1] = sum.y; out[2] = sum.z; out[3] = sum.w; }
}

// Fixed-size dispatch of an expert-parallel layer.  Slot s = (destination rank d, position i) of the send
// buffer holds the i-th pair (in pair order) whose expert lives on rank d, or id -1 if there are fewer.
// One CTA per slot finds its pair by scanning the T*k ids, copies the pair's Q8_1 planes and local expert
// id, and notes the slot for the way back.  Row: [H int8][d_stride f32][int32 id], row_bytes a multiple of 16.
__global__ void __launch_bounds__(128) ep_pack_kernel(const int32_t* topk_idx, const int8_t* x_q, const float* x_d, int d_stride,
                                                      uint8_t* send, int32_t* slot, int T, int k, int H, int experts_per_rank, int cap,
                                                      int row_bytes) {
    __shared__ int s_pair;
    const int s = blockIdx.x, d = s / cap, i = s - d * cap, P = T * k;
    if (threadIdx.x < 32) {
        // warp 0: the i-th pair with destination d, pairs in ascending order
        int found = -1, seen = 0;
        for (int base = 0; base < P && found < 0; base += 32) {
            const int q = base + threadIdx.x;
            const bool hit = q < P && (__ldcg(topk_idx + q) / experts_per_rank) == d;
            const unsigned m = __ballot_sync(0xffffffffu, hit);
            const int c = __popc(m);
            if (seen + c > i) {
                unsigned mm = m;
                for (int r = 0; r < i - seen; ++r) mm &= mm - 1;   // drop the first i - seen hits
                found = base + __ffs(mm) - 1;
            }
            seen += c;
        }
        if (threadIdx.x == 0) s_pair = found;
    }
    __syncthreads();
    const int pair = s_pair;
    uint8_t* row = send + (size_t)s * row_bytes;
    int32_t* idp = reinterpret_cast<int32_t*>(row + H + 4 * d_stride);
    if (pair < 0) {
        if (threadIdx.x == 0) *idp = -1;
        return;
    }
    const int t = pair / k;
    const uint4* sq = reinterpret_cast<const uint4*>(x_q + (size_t)t * H);
    for (int v = threadIdx.x; v < H / 16; v += blockDim.x) reinterpret_cast<uint4*>(row)[v] = sq[v];
    const float* sd = x_d + (size_t)t * d_stride;
    for (int v = threadIdx.x; v < d_stride; v += blockDim.x) reinterpret_cast<float*>(row + H)[v] = sd[v];
    if (threadIdx.x == 0) {
        *idp = __ldcg(topk_idx + pair) - d * experts_per_rank;
        slot[pair] = s;
    }
}

// ---- expert-parallel exchange by peer stores (decode-size batches) -----------------------------
// Instead of handing the packed rows to a collective, the home rank writes every pair's row straight into its owner's
// receive buffer (peer memory over NVLink, plain stores, no multicast), and the owner writes every (home rank, token)
// partial sum straight into the home rank's buffer.  One counter per (buffer, source rank) says how many of the source's
// CTAs have finished writing their part of this call: every CTA adds one with a system-scope release behind its stores,
// the reader waits (acquire) for the full count and takes the counter down again.  A rank cannot be a call ahead of a peer
// on the same buffers (it needs that peer's answer first), so one counter suffices.
// Every wait is bounded; a wait that runs out raises the status bit and the kernel goes on.
// Row: [H int8][d_stride f32][int32 local expert id | -1][int32 token][f32 routing weight], row_bytes a multiple of 16.
// One CTA per slot s = (destination rank d, position i): the i-th pair (in pair order) whose expert lives on rank d goes
// to row rank * cap + i of rank d's receive buffer; slots without a pair get id -1.
__global__ void __launch_bounds__(128) ep_pack_p2p_kernel(const int32_t* topk_idx, const float* topk_w, const int8_t* x_q, const float* x_d,
                                                          int d_stride, uint8_t* const* peer_recv, int32_t* const* peer_flags,
                                                          int rank, int T, int k, int H, int experts_per_rank, int cap, int row_bytes) {
    __shared__ int s_pair;
    const int s = blockIdx.x, d = s / cap, i = s - d * cap, P = T * k;
    if (threadIdx.x < 32) {
        int found = -1, seen = 0;
        for (int base = 0; base < P && found < 0; base += 32) {
            const int q = base + threadIdx.x;
            const bool hit = q < P && (__ldcg(topk_idx + q) / experts_per_rank) == d;
            const unsigned m = __ballot_sync(0xffffffffu, hit);
            const int c = __popc(m);
            if (seen + c > i) {
                unsigned mm = m;
                for (int r = 0; r < i - seen; ++r) mm &= mm - 1;   // drop the first i - seen hits
                found = base + __ffs(mm) - 1;
            }
            seen += c;
        }
        if (threadIdx.x == 0) s_pair = found;
    }
    __syncthreads();
    const int pair = s_pair;
    uint8_t* row = peer_recv[d] + ((size_t)rank * cap + i) * row_bytes;
    int32_t* tail = reinterpret_cast<int32_t*>(row + H + 4 * d_stride);
    if (pair < 0) {
        if (threadIdx.x == 0) tail[0] = -1;
    } else {
        const int t = pair / k;
        const uint4* sq = reinterpret_cast<const uint4*>(x_q + (size_t)t * H);
        for (int v = threadIdx.x; v < H / 16; v += blockDim.x) reinterpret_cast<uint4*>(row)[v] = sq[v];
        const float* sd = x_d + (size_t)t * d_stride;
        for (int v = threadIdx.x; v < d_stride; v += blockDim.x) reinterpret_cast<float*>(row + H)[v] = sd[v];
        if (threadIdx.x == 0) {
            tail[0] = __ldcg(topk_idx + pair) - d * experts_per_rank;
            tail[1] = t;
            reinterpret_cast<float*>(tail)[2] = __ldcg(topk_w + pair);
        }
    }
    // this CTA's stores, then one more on the destination's counter for this rank (the CTA barrier orders every thread's
    // stores before thread 0's release; releases are cumulative): the reader waits for `cap` of them
    __syncthreads();
    if (threadIdx.x == 0) red_release_sys_add(peer_flags[d] + rank, 1);
}

// Owner side, before its kernels read the received rows: wait for every source rank's counter and take it down.
__global__ void ep_wait_flags_kernel(int32_t* flags, int n, int expect, int32_t* status) {
    const int i = threadIdx.x;
    if (i < n) {
        if (!wait_flag(flags + i, expect) && status) atomicOr(status, kStatusWaitTimeout);
        flags[i] = 0;
    }
}

// Owner side, after the down products: for every (source rank s, token t) the routing-weighted sum of the expert rows of
// that token's pairs on this rank, in slot order, written into rank s's buffer at [this rank][t][H]; then this rank's flag
// there.  grid = (world * T, ceil(H / 256)), 256 threads.
__global__ void __launch_bounds__(256) ep_return_p2p_kernel(const float* pair_rows, const uint8_t* recv, int row_bytes, int tail_off,
                                                            float* const* peer_back, int32_t* const* peer_flags, int rank, int T, int cap,
                                                            int H) {
    __shared__ float s_w[64];
    __shared__ int s_slot[64];
    __shared__ int s_n;
    const int s = blockIdx.x / T, t = blockIdx.x - s * T;
    // the slots of source s that carry a pair of token t (at most top_k <= 8 of them), kept in slot order
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int n = 0;
        for (int base = 0; base < cap; base += 32) {
            const int i = base + lane;
            bool hit = false;
            float wgt = 0.0f;
            if (i < cap) {
                const int32_t* tail = reinterpret_cast<const int32_t*>(recv + ((size_t)s * cap + i) * row_bytes + tail_off);
                hit = __ldcg(tail) >= 0 && __ldcg(tail + 1) == t;
                wgt = __ldcg(reinterpret_cast<const float*>(tail) + 2);
            }
            const unsigned m = __ballot_sync(0xffffffffu, hit);
            const int pos = n + __popc(m & ((1u << lane) - 1u));
            if (hit && pos < 64) { s_slot[pos] = s * cap + i; s_w[pos] = wgt; }
            n += __popc(m);
        }
        if (lane == 0) s_n = min(n, 64);
    }
    __syncthreads();
    const int n = s_n;
    const int h = blockIdx.y * 256 + threadIdx.x;
    if (h < H) {
        float sum = 0.0f;
        for (int j = 0; j < n; ++j) sum = fmaf(s_w[j], __ldcg(pair_rows + (size_t)s_slot[j] * H + h), sum);
        peer_back[s][((size_t)rank * T + t) * H + h] = sum;
    }
    __syncthreads();
    if (threadIdx.x == 0) red_release_sys_add(peer_flags[s] + rank, 1);   // the home rank waits for T * gridDim.y of these
}

// Home side: y[t] = sum over owner ranks (ascending) of their partial sums + the sigmoid-gated shared expert.  Every CTA
// waits for the owners' flags; the CTA that finishes last takes them down.  ctr: one int of local scratch.
__global__ void __launch_bounds__(256) ep_finish_p2p_kernel(const float* back, int32_t* flags, int world, int expect, const float* shared_rows,
                                                            const float* sh_logit, float* y, int T, int H, int32_t* ctr, int32_t* status) {
    __shared__ int s_ok;
    if (threadIdx.x == 0) s_ok = 1;
    __syncthreads();
    if (threadIdx.x < world && !wait_flag(flags + threadIdx.x, expect)) s_ok = 0;
    __syncthreads();
    if (!s_ok && threadIdx.x == 0 && status) atomicOr(status, kStatusWaitTimeout);
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < (int64_t)T * H) {
        const int t = (int)(idx / H), h = (int)(idx - (int64_t)t * H);
        float sum = 0.0f;
        for (int o = 0; o < world; ++o) sum += __ldcg(back + ((size_t)o * T + t) * H + h);
        if (shared_rows) {
            const float sh = shared_rows[(size_t)t * H + h];
            if (sh_logit) sum = fmaf(sh, sigmoid_ref(sh_logit[t]), sum);
            else sum = sh + sum;
        }
        y[idx] = sum;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(ctr, 1) == (int)gridDim.x - 1) {
            *ctr = 0;
            for (int o = 0; o < world; ++o) flags[o] = 0;
        }
    }
}

cudaError_t launch_ep_pack_p2p(const int32_t* topk_idx, const float* topk_w, const int8_t* x_q, const float* x_d, int d_stride,
                               uint8_t* const* peer_recv, int32_t* const* peer_flags, int rank, int T, int k, int H,
                               int experts_per_rank, int world, int cap, int row_bytes, cudaStream_t stream) {
    ep_pack_p2p_kernel<<<world * cap, 128, 0, stream>>>(topk_idx, topk_w, x_q, x_d, d_stride, peer_recv, peer_flags, rank, T, k, H,
                                                        experts_per_rank, cap, row_bytes);
    return cudaGetLastError();
}
cudaError_t launch_ep_wait_flags(int32_t* flags, int n, int expect, int32_t* status, cudaStream_t stream) {
    ep_wait_flags_kernel<<<1, 32, 0, stream>>>(flags, n, expect, status);
    return cudaGetLastError();
}
cudaError_t launch_ep_return_p2p(const float* pair_rows, const uint8_t* recv, int row_bytes, int tail_off, float* const* peer_back,
                                 int32_t* const* peer_flags, int rank, int world, int T, int cap, int H, cudaStream_t stream) {
    ep_return_p2p_kernel<<<dim3(world * T, (H + 255) / 256), 256, 0, stream>>>(pair_rows, recv, row_bytes, tail_off, peer_back, peer_flags, rank,
                                                                              T, cap, H);
    return cudaGetLastError();
}
// the home rank's counters reach T * ceil(H / 256) per owner rank
cudaError_t launch_ep_finish_p2p(const float* back, int32_t* flags, int world, const float* shared_rows, const float* sh_logit, float* y,
                                 int T, int H, int32_t* ctr, int32_t* status, cudaStream_t stream) {
    const int64_t n = (int64_t)T * H;
    if (n <= 0) return cudaSuccess;
    ep_finish_p2p_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(back, flags, world, T * ((H + 255) / 256), shared_rows, sh_logit, y, T, H,
                                                                         ctr, status);
    return cudaGetLastError();
}

static size_t route_smem(int TT, int TE) {
    size_t a = (size_t)TT * TE * 256 * sizeof(float);
    size_t b = kDispatchSmemInts * sizeof(int);
    return a > b ? a : b;
}

cudaError_t launch_permute(const RouteParams& p, cudaStream_t stream) {
    if (use_split_dispatch(p) && !p.wait_flags) return launch_dispatch_split(p, false, stream);
    permute_kernel<<<1, 256, (kDispatchSmemInts + kPermuteIdsRoom) * sizeof(int), stream>>>(p);
    return cudaGetLastError();
}

// The routing decision of a layer call in the form the drafter tooling stores it: one byte per (token, slot), slots
// in descending-score order (the "ffn_moe_topk-{L}" tensor, I32 [n_expert_used, n_tokens], narrowed to uint8
// [n_tokens][8]; chimere-dflash/extract/target_daemon.cpp:18-23).  `load` (optional) collects how many pairs each expert
// received: the per-expert load metric.
__global__ void routing_trace_kernel(const int32_t* topk_idx, uint8_t* trace, int32_t* load, int n, int E) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int e = topk_idx[i];
    trace[i] = (uint8_t)e;
    if (load && e >= 0 && e < E) atomicAdd(load + e, 1);
}

cudaError_t launch_routing_trace(const int32_t* topk_idx, uint8_t* trace, int32_t* load, int T, int k, int E, cudaStream_t stream) {
    const int n = T * k;
    if (n <= 0) return cudaSuccess;
    routing_trace_kernel<<<(n + 255) / 256, 256, 0, stream>>>(topk_idx, trace, load, n, E);
    return cudaGetLastError();
}

cudaError_t launch_ep_finish(const float* rows, const int32_t* slot, const float* topk_w, const float* shared_rows, const float* sh_logit,
                             float* y, int T, int H, int k, cudaStream_t stream) {
    const int64_t n = (int64_t)T * (H / 4);   // (H is a multiple of 32)
    if (n <= 0) return cudaSuccess;
    const bool aligned = (((uintptr_t)rows | (uintptr_t)shared_rows | (uintptr_t)y) & 15) == 0;   // (H is a multiple of four: so is every row then)
    return launch_pdl(aligned ? ep_finish_kernel<true> : ep_finish_kernel<false>, dim3((unsigned)((n + 255) / 256)), 256, 0, stream, rows, slot, topk_w,
                      shared_rows, sh_logit, y, T, H, k);
}

// Exact-size dispatch (prefill-size batches): the routing kernel's dispatch has already sorted the pairs by expert, and the
// experts of an owner rank are contiguous, so perm[] lists the pairs grouped by destination.  One CTA per sorted position j
// copies pair perm[j]'s row in the same row format as above and notes slot[pair] = j for the way back.
__global__ void __launch_bounds__(128) ep_pack_sorted_kernel(const int32_t* perm, const int32_t* topk_idx, const int8_t* x_q, const float* x_d,
                                                             int d_stride, uint8_t* send, int32_t* slot, int k, int H, int experts_per_rank,
                                                             int row_bytes) {
    const int j = blockIdx.x, pair = __ldcg(perm + j), t = pair / k;
    const int e = __ldcg(topk_idx + pair);
    uint8_t* row = send + (size_t)j * row_bytes;
    const uint4* sq = reinterpret_cast<const uint4*>(x_q + (size_t)t * H);
    for (int v = threadIdx.x; v < H / 16; v += blockDim.x) reinterpret_cast<uint4*>(row)[v] = sq[v];
    const float* sd = x_d + (size_t)t * d_stride;
    for (int v = threadIdx.x; v < d_stride; v += blockDim.x) reinterpret_cast<float*>(row + H)[v] = sd[v];
    if (threadIdx.x == 0) {
        *reinterpret_cast<int32_t*>(row + H + 4 * d_stride) = e % experts_per_rank;
        slot[pair] = j;
    }
}
cudaError_t launch_ep_pack_sorted(const int32_t* perm, const int32_t* topk_idx, const int8_t* x_q, const float* x_d, int d_stride, uint8_t* send,
                                  int32_t* slot, int T, int k, int H, int experts_per_rank, int row_bytes, cudaStream_t stream) {
    if (T * k <= 0) return cudaSuccess;
    ep_pack_sorted_kernel<<<T * k, 128, 0, stream>>>(perm, topk_idx, x_q, x_d, d_stride, send, slot, k, H, experts_per_rank, row_bytes);
    return cudaGetLastError();
}

cudaError_t launch_ep_pack(const int32_t* topk_idx, const int8_t* x_q, const float* x_d, int d_stride, uint8_t* send, int32_t* slot,
                           int T, int k, int H, int experts_per_rank, int world, int cap, int row_bytes, cudaStream_t stream) {
    ep_pack_kernel<<<world * cap, 128, 0, stream>>>(topk_idx, x_q, x_d, d_stride, send, slot, T, k, H, experts_per_rank, cap, row_bytes);
    return cudaGetLastError();
}

// The tiled product's three launches start to pay where the simple kernel (a CTA per 8 tokens x 8 experts, partials through shared
// memory) fills the GPU more than once: 19.6 against 29 us at 61 x 257 outputs of H = 2048, 32 against 33 at 130 x 257.  From 513 columns on,
// though the row is one kilo-element, 256 experts of H = 1024: 128 tokens 1.15 times the simple kernel's time, 160 0.94, 256 35 us against 41; H = 640: 1.16,
// 0.97, 0.83.  Shorter rows: H = 512, 65536 outputs 0.91 (256 experts) to 1.12 (64), H = 256 0.99 to 1.12.
constexpr int kRouteTileWork = 65536, kRouteTileOutputs = 36864;
static bool route_tiled(const RouteParams& p) {
    const int64_t outputs = (int64_t)p.T * p.E;
    return (outputs * route_nq(p.H) > kRouteTileWork || (p.H > 512 && outputs > kRouteTileOutputs)) && p.scratch && p.H <= 4096 &&
           route_scratch_floats(p.T, p.E, p.H) <= p.scratch_floats;
}
// Tiles of 16 tokens instead of 32 while all of them run at once, two per SM (one where a row has more than 2048 columns, whose rings are then four
// deep: a warp alone on its SM quarter waits for its copies).  Prefill call, us, 32 / 16: 256 experts of H = 2048, 160 tokens 120.6 / 112.8, 256: 137.0 /
// 130.6, 288: 147.0 / 144.0, 384 and 512 (over the line) 166.4 / 168.1, 189.5 / 194.0; 128 of H = 2688, 180 tokens 352.6 / 347.5, 256: 371.9 / 367.4 (372.9 /
// 373.4 with a ring of two), 512 (over the line) 505.8 / 510.3.
template <int NQ, int TA> static int64_t route_tiles(const RouteParams& p) {
    using R = RouteTile<NQ, TA>;
    return (int64_t)((p.E + R::kExp - 1) / R::kExp) * ((p.T + R::kTok - 1) / R::kTok);
}
template <int NQ, int TA>
static cudaError_t launch_route_tile(const RouteParams& p, cudaStream_t stream) {
    using R = RouteTile<NQ, TA>;
    static bool attr_done[64] = {};
    const cudaError_t e = max_smem_once(route_tile_kernel<NQ, TA>, (int)R::kSmem, attr_done);
    if (e != cudaSuccess) return e;
    return launch_pdl(route_tile_kernel<NQ, TA>, dim3((p.E + R::kExp - 1) / R::kExp, (p.T + R::kTok - 1) / R::kTok), 256, R::kSmem, stream, p);
}
template <int NQ>
static cudaError_t launch_route_tiles(const RouteParams& p, cudaStream_t stream) {
    const bool half = route_tiles<NQ, 2>(p) <= (NQ > 2 ? 1 : 2) * sm_count();
    cudaError_t e = launch_pdl(route_prep_kernel<NQ>, dim3(p.T + p.E), 256, 0, stream, p);
    if (e == cudaSuccess) e = half ? launch_route_tile<NQ, 2>(p, stream) : launch_route_tile<NQ, 4>(p, stream);
    if (e != cudaSuccess) return e;
    const bool split = use_split_dispatch(p);
    // (four tokens per warp at most: with fewer experts per token the counts are a launch of their own)
    const bool counted = split && p.top_k >= 4;
    const int tokens = counted ? dispatch_tokens(p.top_k) : 8;
    e = counted ? launch_pdl(route_topk_kernel, dim3(dispatch_chunks(p.T, p.top_k)), 256, (256 + kDispatchChunk) * 4, stream, p, p.dispatch_scratch, tokens)
                : launch_pdl(route_topk_kernel, dim3((p.T + 7) / 8), 256, (kDispatchSmemInts + kTopkIdsRoom) * 4, stream, p, (int32_t*)nullptr, split ? 0 : tokens);
    return e == cudaSuccess && split ? launch_dispatch_split(p, counted, stream) : e;
}

bool route_norm_runs(const RouteParams& p) { return p.T <= 4 && p.H <= 256 * 12; }
template <int TT>
static cudaError_t launch_route_norm_t(const RouteParams& p, const float* hidden, const float* residual, const float* weight, float eps, cudaStream_t stream) {
    const dim3 grid((p.E + (p.shexp_gate_w ? 1 : 0) + 1) / 2);
    if (p.H <= 256 * 8) return launch_pdl(route_norm_kernel<TT, 8>, grid, 256, 0, stream, p, hidden, residual, weight, eps);
    return launch_pdl(route_norm_kernel<TT, 12>, grid, 256, 0, stream, p, hidden, residual, weight, eps);
}
cudaError_t launch_route_norm(const RouteParams& p, const float* hidden, const float* residual, const float* weight, float eps, cudaStream_t stream) {
    return p.T == 1 ? launch_route_norm_t<1>(p, hidden, residual, weight, eps, stream)
                    : p.T == 2 ? launch_route_norm_t<2>(p, hidden, residual, weight, eps, stream) : launch_route_norm_t<4>(p, hidden, residual, weight, eps, stream);
}

cudaError_t launch_route(const RouteParams& p, cudaStream_t stream) {
    const int nrows = p.E + (p.shexp_gate_w ? 1 : 0);
    const int ttiles8 = (p.T + 7) / 8;
    // One and two tokens: pairs of router rows per CTA, sized for so many tokens (route entry of 128 experts, one token of 2048 columns 7.3 -> 5.3 us,
    // of 2688 7.9 -> 5.7, against the forms for eight).  Up to 32, few experts: a row per CTA, up to 3072 columns in flight at once, as long as that is one
    // CTA per SM (64 experts of H = 2048, 8 tokens 9.6 -> 9.1 us, but 24 tokens 10.9 -> 11.7).
    if (p.T <= 2) {
        constexpr int TE = 2;
        const dim3 grid((nrows + TE - 1) / TE);
        return p.T == 1 ? launch_pdl(route_kernel<1, TE>, grid, 256, route_smem(1, TE), stream, p) : launch_pdl(route_kernel<2, TE>, grid, 256, route_smem(2, TE), stream, p);
    } else if (p.T <= 32 && nrows * ttiles8 <= sm_count()) {
        constexpr int TT = 8, TE = 1;
        return launch_pdl(route_kernel<TT, TE>, dim3(nrows, (p.T + TT - 1) / TT), 256, route_smem(TT, TE), stream, p);
    } else if (p.T <= 32) {
        constexpr int TT = 8, TE = 2;
        dim3 grid((nrows + TE - 1) / TE, (p.T + TT - 1) / TT);
        return launch_pdl(route_kernel<TT, TE>, grid, 256, route_smem(TT, TE), stream, p);
    } else if (route_tiled(p)) {
        switch (route_nq(p.H)) {
            case 1: return launch_route_tiles<1>(p, stream);
            case 2: return launch_route_tiles<2>(p, stream);
            case 3: return launch_route_tiles<3>(p, stream);
            default: return launch_route_tiles<4>(p, stream);
        }
    } else {
        constexpr int TT = 8, TE = 8;
        const unsigned rtiles = (nrows + TE - 1) / TE, ttiles = (p.T + TT - 1) / TT;
        static bool attr_done[64] = {}, attr_done_x[64] = {};
        if (ttiles > 65535) {
            cudaError_t e = max_smem_once(route_kernel<TT, TE, true>, (int)route_smem(TT, TE), attr_done_x);
            if (e != cudaSuccess) return e;
            route_kernel<TT, TE, true><<<dim3(ttiles, rtiles), 256, route_smem(TT, TE), stream>>>(p);
            return cudaGetLastError();
        }
        cudaError_t e = max_smem_once(route_kernel<TT, TE>, (int)route_smem(TT, TE), attr_done);
        if (e != cudaSuccess) return e;
        route_kernel<TT, TE><<<dim3(rtiles, ttiles), 256, route_smem(TT, TE), stream>>>(p);
    }
    return cudaGetLastError();
}

}  // namespace chimere

// ------------------------------------------------------------------------------------------
// Routing without any allocation by anyone: chimere_b200_moe_route_noalloc.
//
// Some hosts of this library cannot hand it scratch memory.  A serving process that gave all device
// memory to its own pool at start-up (the reference's server sizes every buffer once, at model
// load), or a caller already inside a region where cudaMalloc is not permitted, has the token rows
// and somewhere to put the routing result, but no spare arena and no way to get one.  For them the
// routing step's scratch lives in the library image itself: one fixed array per GPU, reserved when
// the library is loaded on that GPU and held until the process ends.
//
// In host code the array's name is only a handle, not a device address, so the address is looked
// up once per device with cudaGetSymbolAddress (with that device current) and cached.  The first
// call on a device does this look-up; make that first call outside any stream capture.
// Every call on a device shares the one array: calls that overlap on the GPU (two streams, two
// threads) race.  Nothing here calls cudaMalloc, cudaFree or a library routine that allocates.
namespace chimere {

constexpr int kNoAllocMaxT = 64;        // tokens per call
constexpr int kNoAllocMaxH = 4096;      // hidden size
constexpr size_t kNoAllocCounters = 0;                                                        // 1 KiB of integer scratch
constexpr size_t kNoAllocLogits = 1024;                                                       // [T][256] f32
constexpr size_t kNoAllocShLogit = kNoAllocLogits + (size_t)kNoAllocMaxT * kMaxExperts * 4;   // [T] f32
constexpr size_t kNoAllocXq8 = kNoAllocShLogit + 256;                                         // [T][H/32][36]
constexpr size_t kNoAllocXq = kNoAllocXq8 + (size_t)kNoAllocMaxT * (kNoAllocMaxH / 32) * kQ81Bytes;
constexpr size_t kNoAllocXd = kNoAllocXq + (size_t)kNoAllocMaxT * kNoAllocMaxH;               // [T][H/32] f32
constexpr size_t kNoAllocPerm = kNoAllocXd + (size_t)kNoAllocMaxT * (kNoAllocMaxH / 32) * 4;  // [T*8] i32
constexpr size_t kNoAllocOffsets = kNoAllocPerm + (size_t)kNoAllocMaxT * kMaxTopK * 4;        // [257] i32
constexpr size_t kNoAllocList = kNoAllocOffsets + 1280;                                       // work list
constexpr int kNoAllocEntries = kMaxExperts + kNoAllocMaxT * kMaxTopK + kNoAllocMaxT;
constexpr size_t kNoAllocBytes = kNoAllocList + (size_t)(kListHeader + kListEntry * kNoAllocEntries) * 4 + 256;

static __device__ __align__(256) unsigned char g_route_scratch[kNoAllocBytes];   // ~680 KiB per GPU

}  // namespace chimere

extern "C" int chimere_b200_moe_route_noalloc(const chimere_moe_layer* w, const float* d_x, int T, int32_t* d_topk_idx,
                                              float* d_topk_w, cudaStream_t stream) {
    using namespace chimere;
    if (!w || !d_x || !d_topk_idx || !d_topk_w || !w->router_w) return -1;
    if (w->H <= 0 || w->H % 32 || w->E <= 0 || w->top_k <= 0 || w->top_k > w->E || T <= 0) return -2;
    if (w->route_mode != CHIMERE_ROUTE_SOFTMAX_RENORM && w->route_mode != CHIMERE_ROUTE_SIGMOID_NORM_SCALE) return -2;
    // larger than the built-in scratch was sized for: use chimere_b200_moe_route with a workspace instead
    if (T > kNoAllocMaxT || w->H > kNoAllocMaxH || w->E > kMaxExperts || w->top_k > kMaxTopK) return -7;

    // once per device, with that device current: the array's device address
    static unsigned char* s_base[64] = {nullptr};
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return -100 - (int)e;
    if (dev < 0 || dev >= 64) return -2;
    if (!s_base[dev]) {
        // the look-up is not a stream operation and must not happen while `stream` is being captured
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(stream, &cap) == cudaSuccess && cap != cudaStreamCaptureStatusNone) return -8;
        unsigned char* ptr = nullptr;
        e = cudaGetSymbolAddress((void**)&ptr, g_route_scratch);
        if (e != cudaSuccess || !ptr) return -100 - (int)e;
        s_base[dev] = ptr;
    }
    unsigned char* base = s_base[dev];

    // the integer scratch must start at zero; everything else is fully rewritten by the kernel
    e = cudaMemsetAsync(base + kNoAllocCounters, 0, 1024, stream);
    if (e != cudaSuccess) return -100 - (int)e;

    RouteParams p{};
    p.T = T; p.H = w->H; p.E = w->E; p.top_k = w->top_k; p.route_mode = w->route_mode;
    p.has_shared = w->F_s > 0;
    p.route_scale = w->route_scale;
    p.x = d_x; p.router_w = w->router_w; p.router_bias = w->router_bias;
    p.shexp_gate_w = (w->F_s > 0) ? w->shexp_gate_w : nullptr;
    p.counters = (int32_t*)(base + kNoAllocCounters);
    p.router_logits = (float*)(base + kNoAllocLogits);
    p.sh_gate_logit = (float*)(base + kNoAllocShLogit);
    p.x_q8 = base + kNoAllocXq8;
    p.x_soa_q = (int8_t*)(base + kNoAllocXq);
    p.x_soa_d = (float*)(base + kNoAllocXd);
    p.x_soa_d_stride = (w->H / 32 + 3) & ~3;
    p.perm = (int32_t*)(base + kNoAllocPerm);
    p.offsets = (int32_t*)(base + kNoAllocOffsets);
    p.group_list = (int32_t*)(base + kNoAllocList);
    p.list_capacity = kNoAllocEntries;
    p.topk_idx = d_topk_idx;   // results go straight to the caller's buffers
    p.topk_w = d_topk_w;
    e = launch_route(p, stream);
    return e == cudaSuccess ? 0 : -100 - (int)e;
}
