// routing.cuh -- a token's top-k and the dispatch of a batch's (token, expert) pairs: steps of the router's last CTA (router.cu) and,
// in batches whose pairs are work items of their own, of the expert kernels themselves (pairs.cu).
#pragma once
#include "common.cuh"
#include "kernels.h"

namespace chimere {

// One token's scores -> top-k, by one warp; lane l owns experts l, l+32, ...  Returns lane j's slot j: expert and combine weight.  With
// fewer rounds than top_k only the ids of the first `rounds` slots are meant.
struct TopkSlot { int id; float w; };
__device__ __forceinline__ TopkSlot topk_select(const RouteParams& p, const float* logit_row, int lane, int rounds) {
    const int E = p.E, k = p.top_k;
    // (No branches on a lane's data in the ordinary path: each would hold up the shuffles and exponentials behind it.)
    float v[8], pr[8];
    uint32_t there[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        there[i] = (uint32_t)((lane + 32 * i - E) >> 31);   // all ones for an expert, 0 beyond the last
        v[i] = -1.0e30f;
        if (there[i]) v[i] = __ldcg(logit_row + lane + 32 * i);
    }
    if (p.route_mode == CHIMERE_ROUTE_SOFTMAX_RENORM) {
        // largest logit: integers that order like the floats (a NaN comes out on top, and makes the sum one either way)
        auto ordered = [](float x) { const int b = __float_as_int(x); return b ^ (int)((uint32_t)(b >> 31) >> 1); };
        int top = ordered(v[0]);
#pragma unroll
        for (int i = 1; i < 8; ++i) top = max(top, ordered(v[i]));
        top = __reduce_max_sync(0xffffffffu, top);
        const float mx = __int_as_float(top ^ (int)((uint32_t)(top >> 31) >> 1));
        float ev[8], least = 1.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t bits = __float_as_uint(expf(v[i] - mx));
            ev[i] = __uint_as_float(bits & there[i]);
            least = fminf(least, __uint_as_float((bits & there[i]) | (0x3F800000u & ~there[i])));   // (a NaN passes by here, and shows in the sum)
        }
        // tree256's order: the values 128 and 64 and 32 elements apart are this lane's own
        float sum = ((ev[0] + ev[4]) + (ev[2] + ev[6])) + ((ev[1] + ev[5]) + (ev[3] + ev[7]));
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, s);
        sum = __shfl_sync(0xffffffffu, sum, 0);
        if (__all_sync(0xffffffffu, least > 1e-25f && sum < 1e9f)) {   // (no quotient near the subnormals)
            const float r = __frcp_rn(sum);
#pragma unroll
            for (int i = 0; i < 8; ++i) pr[i] = div_by_recip(ev[i], sum, r);   // the division operator's bits
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) pr[i] = (sum > 0.0f) ? (ev[i] / sum) : (1.0f / (float)E);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) pr[i] = __frcp_rn(1.0f + expf(-v[i]));   // (correctly rounded, as 1.0f / ...)
    }
    // Selection on integer keys: probabilities are >= 0, so their bit patterns order like the values; key 0 = not available (beyond E,
    // or already taken).  One warp-wide max and one warp-wide min per slot (redux.sync): the largest value wins, equal values go to the
    // lowest index, like a strict-greater scan from index 0.  A round is about 100 cycles; it is a loop because this code runs
    // once per launch, and fetching it unrolled takes longer than running it (ranks from 32 shuffles at once: 4 400 cycles cold against 2 800).
    uint32_t key[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) key[i] = (__float_as_uint(pr[i]) + 1u) & there[i];
    float wsum = 0.0f;
    float wsel = 0.0f;  // lane j keeps the weight of slot j
    int isel = 0;
#pragma unroll 1
    for (int j = 0; j < rounds; ++j) {
        const uint32_t m = __reduce_max_sync(0xffffffffu, max(max(max(key[0], key[1]), max(key[2], key[3])), max(max(key[4], key[5]), max(key[6], key[7]))));
        uint32_t c[8];   // where this lane holds the maximum
#pragma unroll
        for (int i = 0; i < 8; ++i) c[i] = key[i] == m ? (uint32_t)(lane + 32 * i) : 0xffffu;
        const uint32_t bi = __reduce_min_sync(0xffffffffu, min(min(min(c[0], c[1]), min(c[2], c[3])), min(min(c[4], c[5]), min(c[6], c[7]))));
        const float bv = __uint_as_float(m - 1u);
        wsum += bv;
        wsel = lane == j ? bv : wsel;
        isel = lane == j ? (int)bi : isel;
#pragma unroll
        for (int i = 0; i < 8; ++i) key[i] = bi == (uint32_t)(lane + 32 * i) ? 0u : key[i];
    }
    if (lane < k) {
        if (wsum > 0.0f) {
            const float inv = __frcp_rn(wsum);   // (correctly rounded, as 1.0f / wsum)
            wsel = wsel * inv;
        }
        if (p.route_mode != CHIMERE_ROUTE_SOFTMAX_RENORM || p.route_scale != 1.0f) wsel = wsel * p.route_scale;
    }
    return TopkSlot{isel, wsel};
}
__device__ __forceinline__ void topk_warp(const RouteParams& p, const float* logit_row, int t, int lane, int* ids_out) {
    const TopkSlot s = topk_select(p, logit_row, lane, p.top_k);
    if (lane < p.top_k) {
        p.topk_idx[(size_t)t * p.top_k + lane] = s.id;
        p.topk_w[(size_t)t * p.top_k + lane] = s.w;
        if (ids_out) ids_out[lane] = s.id;
    }
}

// Stable counting sort of the T*k pairs by expert, plus the GEMV work list.  One CTA of 256.
// s_ids: the T*k expert ids in shared memory if the caller has them there (else they are read from p.topk_idx).
// Each warp takes one contiguous eighth of the pairs: it counts its pairs per expert, the counts are turned into
// every warp's first position within every expert, and the warp places its pairs in order; so the only CTA
// barriers are between those steps, however many pairs there are.  The work entries are then filled by all
// threads (entry -> expert by bisection of the entry offsets).
constexpr int kDispatchSmemInts = 256 + 256 + 2048 + 32 + 288 + 1024;
// The dispatch step is written for 256 threads; in a larger CTA only the first 256 threads call it, so its meeting
// point is a named barrier of those threads (in a CTA of 256 it is the same as a CTA-wide barrier).
__device__ __forceinline__ void dispatch_sync() { asm volatile("bar.sync 2, 256;" ::: "memory"); }
// ids_room: ints of shared memory behind the kDispatchSmemInts of scratch; if the ids fit there they are fetched
// once, all loads in flight together, instead of one dependent load per step of the two passes.
// The same result for at most 32 pairs whose ids are in shared memory (a decode batch of up to four tokens): every thread counts directly --
// pair q its position (ids below its own, equal ids before it), thread e the offset of expert e -- and the work entries
// come from the sorted ids by two ballots.  Two barriers instead of six and no scratch to clear: a third of the time.
constexpr int kSmallDispatchPairs = 32;   // (at 64 pairs the direct counting is no faster than the general form)
__device__ __forceinline__ void build_dispatch_small(const RouteParams& p, int* smem_i, const int* s_ids) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int E = p.E, P = p.T * p.top_k;
    int* s_sid = smem_i;          // [64] expert ids in sorted order (room for two warps of positions)
    int* s_perm = smem_i + 64;    // [64] the permutation
    const int gt = p.group > 0 ? p.group : kMaxGroupTokens;
    int* s_lead = smem_i + 128;   // [2] distinct experts among sorted positions 0..31 / 32..63
    const int my_e = tid < P ? s_ids[tid] : -1;
    const bool valid = my_e >= 0 && my_e < E;
    int below_tid = 0, below_mine = 0, before_me = 0, total = 0;
    for (int q = 0; q < P; ++q) {
        const int e = s_ids[q];                      // (the same address in every thread: a broadcast)
        const bool v = e >= 0 && e < E;
        total += v;
        below_tid += v && e < tid;
        below_mine += v && e < my_e;
        before_me += q < tid && e == my_e;
    }
    if (tid < E) p.offsets[tid] = below_tid;
    if (tid == 0) p.offsets[E] = total;
    if (valid) {
        const int pos = below_mine + before_me;
        p.perm[pos] = tid;
        s_perm[pos] = tid;
        s_sid[pos] = my_e;
    }
    // shared-expert entries first (all tokens, identity order), as in the general form
    const int sgt = shared_group_tokens(p.T);
    const int nsh = p.has_shared ? (p.T + sgt - 1) / sgt : 0;
    const int nsh_listed = p.list_mode == 2 ? 0 : nsh;
    for (int i = tid; i < nsh_listed; i += 256) {
        int* ent = p.group_list + kListHeader + kListEntry * i;
        const int t0 = i * sgt, mm = min(sgt, p.T - t0);
        ent[0] = -1; ent[1] = t0; ent[2] = mm; ent[3] = 0;
        for (int j = 0; j < kMaxGroupTokens; ++j) ent[4 + j] = j < mm ? p.T * p.top_k + t0 + j : 0;
    }
    dispatch_sync();
    // sorted position tid starts a new expert?  (warps 0 and 1 hold the 64 positions)
    unsigned lead = 0u;
    if (warp < 2) {
        // (entry starts: every gt-th pair of an expert, gt a power of two; an expert has at most T <= 4 pairs here.  One pair per
        // entry needs no look at the neighbours: this is on the chain of a single token's layer)
        int rank = 0;
        if (gt > 1) while (rank < tid && tid < total && s_sid[tid - rank - 1] == s_sid[tid]) ++rank;
        const bool first = tid < total && (rank & (gt - 1)) == 0;
        lead = __ballot_sync(0xffffffffu, first);
        if (lane == 0) s_lead[warp] = __popc(lead);
    }
    dispatch_sync();
    const int total_routed = p.list_mode != 0 ? 0 : s_lead[0] + s_lead[1];
    if (tid == 0) {
        p.group_list[0] = total_routed + nsh_listed;
        p.group_list[1] = total_routed;
        p.group_list[2] = nsh_listed;
        p.group_list[3] = 0;
    }
    if (warp < 2 && total_routed > 0 && ((lead >> lane) & 1u)) {
        const int idx = __popc(lead & ((1u << lane) - 1u)) + (warp == 1 ? s_lead[0] : 0);
        const int e = s_sid[tid];
        int mm = 1;
        while (mm < gt && tid + mm < total && s_sid[tid + mm] == e) ++mm;
        int* ent = p.group_list + kListHeader + kListEntry * (nsh + idx);
        ent[0] = e; ent[1] = tid; ent[2] = mm; ent[3] = 0;
        for (int j = 0; j < kMaxGroupTokens; ++j) ent[4 + j] = j < mm ? s_perm[tid + j] : 0;
    }
}

__device__ __forceinline__ void build_dispatch(const RouteParams& p, int* smem_i, const int* s_ids, int ids_room) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int E = p.E, P = p.T * p.top_k;
    if (s_ids && P <= kSmallDispatchPairs && p.T <= kMaxGroupTokens) { build_dispatch_small(p, smem_i, s_ids); return; }
    if (!s_ids && P <= ids_room) {
        int* stage = smem_i + kDispatchSmemInts;
        const int istr0 = p.idx_stride > 1 ? p.idx_stride : 1;
        for (int q = tid; q < P; q += 256) stage[q] = __ldcg(p.topk_idx + (size_t)q * istr0);
        s_ids = stage;   // visible after the barrier below
    }
    int* hist = smem_i;               // [256] pairs per expert
    int* cursor = smem_i + 256;       // [256] first position of each expert
    int* warp_cnt = smem_i + 512;     // [8][256] per warp: pairs of each expert, then the warp's next position within it
    int* scan = smem_i + 2560;        // [32]
    int* ent_base = smem_i + 2592;    // [257] first routed entry of each expert, [256] = their number
    int* s_perm = smem_i + 2880;      // [1024] copy of the permutation when it is that short
    const bool perm_in_smem = P <= 1024;
    for (int i = tid; i < 2048; i += 256) warp_cnt[i] = 0;
    dispatch_sync();
    // ids outside [0, E) mark pairs that are not there (padding of a fixed-size exchange): they get no work
    const int istr = p.idx_stride > 1 ? p.idx_stride : 1;
    const int chunk = (((P + 7) >> 3) + 31) & ~31;
    const int q0 = min(P, warp * chunk), q1 = min(P, q0 + chunk);
    for (int base = q0; base < q1; base += 32) {
        const int q = base + lane;
        int e = q < q1 ? (s_ids ? s_ids[q] : __ldcg(p.topk_idx + (size_t)q * istr)) : -1;
        const bool valid = e >= 0 && e < E;
        if (!valid) e = 0x40000000 + lane;
        const unsigned same = __match_any_sync(0xffffffffu, e);
        if (valid && (same & ((1u << lane) - 1u)) == 0u) warp_cnt[warp * 256 + e] += __popc(same);
        __syncwarp();
    }
    dispatch_sync();
    // thread = expert: its pair count, and where each warp's pairs start within it
    int cnt = 0;
    if (tid < E) {
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            const int t = warp_cnt[w * 256 + tid];
            warp_cnt[w * 256 + tid] = cnt;
            cnt += t;
        }
    }
    hist[tid] = cnt;
    // exclusive scans over the experts: pair offsets and work-entry offsets
    const int gt = p.group > 0 ? p.group : kMaxGroupTokens;
    const int nent = (cnt + gt - 1) / gt;
    int incl_c = cnt, incl_n = nent;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, incl_c, s), b = __shfl_up_sync(0xffffffffu, incl_n, s);
        if (lane >= s) { incl_c += a; incl_n += b; }
    }
    if (lane == 31) { scan[warp] = incl_c; scan[8 + warp] = incl_n; }
    dispatch_sync();
    int base_c = 0, base_n = 0;
    for (int w = 0; w < warp; ++w) { base_c += scan[w]; base_n += scan[8 + w]; }
    const int off = base_c + incl_c - cnt;      // exclusive
    const int ent0 = base_n + incl_n - nent;
    cursor[tid] = off;
    ent_base[tid] = ent0;
    if (tid < E) p.offsets[tid] = off;
    if (tid == 255) {
        p.offsets[E] = base_c + incl_c;  // tid 255 holds the inclusive total (cnt = 0 beyond E)
        ent_base[256] = base_n + incl_n;
    }
    int total_routed = 0;
    for (int w = 0; w < 8; ++w) total_routed += scan[8 + w];
    // shared-expert entries first (all tokens, identity order), then the routed ones
    const int sgt = shared_group_tokens(p.T);
    const int nsh = p.has_shared ? (p.T + sgt - 1) / sgt : 0;
    if (p.list_mode != 0) total_routed = 0;
    if (nsh + total_routed > p.list_capacity) {   // (never, if the workspace was made for this layer and batch)
        total_routed = max(0, p.list_capacity - nsh);
        if (tid == 0 && p.status) atomicOr(p.status, kStatusListFull);
    }
    for (int i = tid; i < (p.list_mode == 2 ? 0 : nsh); i += 256) {
        int* ent = p.group_list + kListHeader + kListEntry * i;
        const int t0 = i * sgt, mm = min(sgt, p.T - t0);
        ent[0] = -1; ent[1] = t0; ent[2] = mm; ent[3] = 0;
        for (int j = 0; j < kMaxGroupTokens; ++j) ent[4 + j] = j < mm ? p.T * p.top_k + t0 + j : 0;
    }
    if (tid == 0) {
        const int nsh_listed = p.list_mode == 2 ? 0 : nsh;
        p.group_list[0] = total_routed + nsh_listed;
        p.group_list[1] = total_routed;
        p.group_list[2] = nsh_listed;
        p.group_list[3] = 0;
    }
    dispatch_sync();   // cursor and the warps' first positions are in place
    // stable placement: each warp walks its pairs in order
    for (int base = q0; base < q1; base += 32) {
        const int q = base + lane;
        int e = q < q1 ? (s_ids ? s_ids[q] : __ldcg(p.topk_idx + (size_t)q * istr)) : -1;
        const bool valid = e >= 0 && e < E;
        if (!valid) e = 0x40000000 + lane;
        const unsigned same = __match_any_sync(0xffffffffu, e);
        const int rank = __popc(same & ((1u << lane) - 1u));
        if (valid) {
            const int pos = cursor[e] + warp_cnt[warp * 256 + e] + rank;
            p.perm[pos] = q;
            if (perm_in_smem) s_perm[pos] = q;
        }
        __syncwarp();
        if (valid && rank == 0) warp_cnt[warp * 256 + e] += __popc(same);
        __syncwarp();
    }
    dispatch_sync();
    // the routed entries with their pair rows (perm was written by this CTA: visible after the barrier above)
    for (int idx = tid; idx < total_routed; idx += 256) {
        int lo = 0, hi = 256;   // ent_base[lo] <= idx < ent_base[hi]
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (ent_base[mid] <= idx) lo = mid; else hi = mid;
        }
        const int e = lo, i = idx - ent_base[e], c = hist[e], o = cursor[e];
        const int mm = min(gt, c - i * gt);
        int* ent = p.group_list + kListHeader + kListEntry * (nsh + idx);
        ent[0] = e;
        ent[1] = o + i * gt;
        ent[2] = mm;
        ent[3] = 0;
        for (int j = 0; j < kMaxGroupTokens; ++j)
            ent[4 + j] = j < mm ? (perm_in_smem ? s_perm[o + i * gt + j] : p.perm[o + i * gt + j]) : 0;
    }
}

}  // namespace chimere
