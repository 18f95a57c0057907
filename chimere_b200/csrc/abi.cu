// abi.cu -- host side of the library: the C ABI declared in include/chimere_b200_moe.h.
//
// The layer-level entries are the C++ counterpart of the reference's Rust orchestration
// (forward_moe_cudarc_with_cache, chimere-server/src/qwen35_model/moe_ffn.rs:1081-1768, and its
// scratch owner GgmlGpuBuffers, src/kernels/ggml_gpu.rs:292-407): they validate, lay the
// caller's arena out, and enqueue three kernels per decode call (up to nine where the grouped GEMM takes
// part, up to eleven in prefill).  Nothing here allocates device memory or synchronises, except chimere_b200_moe_forward_host which waits for its stream.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "kernels.h"
#include "tiled.cuh"

using namespace chimere;

namespace {

inline size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }

inline bool type_ok(int t) { return t == CHIMERE_TYPE_Q4_0 || t == CHIMERE_TYPE_Q8_0 || t == CHIMERE_TYPE_IQ3_S; }
inline int type_cols_multiple(int t) { return t == CHIMERE_TYPE_IQ3_S ? 256 : 32; }

inline bool kquant_type(int t) { return t == CHIMERE_TYPE_Q4_K || t == CHIMERE_TYPE_Q5_K || t == CHIMERE_TYPE_Q6_K; }
// A layer whose shared expert is kept in K-quant super-blocks (the production files: Q5_K, moe_ffn.rs:1597-1650).  Its routed
// experts run as a layer without a shared expert; the shared expert follows as plain GEMVs on the raw blocks
// (kshared_chain below), which is how the reference runs it (three GEMV calls, an activation, the sigmoid-gated add).
inline bool kshared(const chimere_moe_layer* w) { return w && w->F_s > 0 && kquant_type(w->type_sh_up); }
inline chimere_moe_layer routed_only(const chimere_moe_layer* w) {
    chimere_moe_layer r = *w;
    r.F_s = 0; r.sh_gate = nullptr; r.sh_up = nullptr; r.sh_down = nullptr;
    r.type_sh_gate = r.type_sh_up = r.type_sh_down = 0;
    return r;   // (keeps shexp_gate_w: the router still computes the gate logit)
}

// ... and whether that shared expert can go through the grouped GEMM (prefill-size batches): all three matrices Q4_K or Q5_K
// (Q6_K has a scale per 16 weights, the MMA's blocks are 32 wide), rows of whole rounds of 32 blocks, gated, read by words.
inline bool kshared_gemm(const chimere_moe_layer* w) {
    auto ok = [](int t) { return t == CHIMERE_TYPE_Q4_K || t == CHIMERE_TYPE_Q5_K; };
    return kshared(w) && w->H % 1024 == 0 && w->act == CHIMERE_ACT_SWIGLU && ok(w->type_sh_gate) && ok(w->type_sh_up) && ok(w->type_sh_down) &&
           (((uintptr_t)w->sh_gate | (uintptr_t)w->sh_up | (uintptr_t)w->sh_down) & 3) == 0;
}

int validate_layer(const chimere_moe_layer* w) {
    if (!w) return -1;
    if (kshared(w)) {
        const bool dual_k = w->act == CHIMERE_ACT_SWIGLU;
        if (!kquant_type(w->type_sh_down) || (dual_k && !kquant_type(w->type_sh_gate))) return -3;
        if (w->H % 256 || w->F_s % 256) return -2;
        if (!w->sh_up || !w->sh_down || (dual_k && !w->sh_gate)) return -1;
        // the shared expert's f32 rows and Q8_1 intermediates borrow the routed pairs' areas of the workspace
        if (2 * (int64_t)w->F_s > (int64_t)w->top_k * w->H || (int64_t)w->F_s > (int64_t)w->top_k * w->F) return -2;
        const chimere_moe_layer r = routed_only(w);
        return validate_layer(&r);
    }
    if (w->H <= 0 || w->E <= 0 || w->E > kMaxExperts || w->F <= 0 || w->F_s < 0) return -2;
    if (w->top_k <= 0 || w->top_k > kMaxTopK || w->top_k > w->E) return -2;
    if (w->H % 32 || w->F % 32 || w->F_s % 32) return -2;
    if (w->layout != CHIMERE_LAYOUT_GGML && w->layout != CHIMERE_LAYOUT_TILED32) return -2;
    if (w->layout == CHIMERE_LAYOUT_TILED32 && w->H % 128) return -2;   // Q8_1 input rows must be 16-byte multiples
    if (w->route_mode != CHIMERE_ROUTE_SOFTMAX_RENORM && w->route_mode != CHIMERE_ROUTE_SIGMOID_NORM_SCALE) return -2;
    if (w->act != CHIMERE_ACT_SWIGLU && w->act != CHIMERE_ACT_RELU2) return -2;
    const bool dual = w->act == CHIMERE_ACT_SWIGLU;
    if (!type_ok(w->type_up) || !type_ok(w->type_down) || (dual && !type_ok(w->type_gate))) return -3;
    if (dual && w->type_gate != w->type_up) return -3;  // gate and up rows are streamed by one kernel instance
    if (w->H % type_cols_multiple(w->type_up) || w->F % type_cols_multiple(w->type_down)) return -2;
    if (!w->router_w || !w->up_exps || !w->down_exps || (dual && !w->gate_exps)) return -1;
    if (w->F_s > 0) {
        if (!type_ok(w->type_sh_up) || !type_ok(w->type_sh_down) || (dual && !type_ok(w->type_sh_gate))) return -3;
        if (dual && w->type_sh_gate != w->type_sh_up) return -3;
        if (w->H % type_cols_multiple(w->type_sh_up) || w->F_s % type_cols_multiple(w->type_sh_down)) return -2;
        if (!w->sh_up || !w->sh_down || (dual && !w->sh_gate)) return -1;
    }
    return 0;
}

// Packed experts (Q4_0, IQ3_S) in the decode entry: up to pair_batch()'s line every (token, expert) pair is an item of its own (pairs.cu; the work
// list where those kernels do not take the layer), which reads an expert once per pair, from L2 behind the first; above it 16 pairs of an
// expert share a tile (mma_tiles.cu), which costs as much with one pair as with eight.  us per layer, pairs / tiles:
//   256 experts of 512 x 2048, top 8, uniform routing: 32 tokens 81 / 111, 40: 101 / 127; skewed: 20: 49 / 47, 40: 90 / 62
//   128 of 1856 x 2688, top 6: 8 tokens 88 / 101, 12: 121 / 122, 16: 159 / 142, 24 (on the GEMM) 189 / 180
// (Before: 40 tokens 115 and 104, 64 tokens 192 and 145, now on the tiles 145 and 70.)  The best line depends on the routing, which the host does
// not know: this one is where neither is slower than the work list's entries of one or two pairs were.
// A call of the tiles has some 14 us that one of the pairs has not (dispatch, combine, longer chains), and small layers or few experts have nothing
// to set against it: what the pairs read again comes from L2 in less.  So whatever the pairs per expert, pairs while they read no more
// weights again than this (uniform routing taken for it).  us, list / tiles / pairs:
//   8 experts of 512 x 2048 top 2: 8 tokens (50M) 22.5 / 31.7 / 19.7, 24 (198M) 37 / 38 / 32, 32 (274M) 41 / 38 / 39, 40 (349M) 65 / 54 / 60
//   64 of 512 x 2048 top 8: 12 tokens (176M) 45 / 55 / 35, 16 (272M) 54 / 58 / 43;   of 256 x 1024: 40 (232M) 50 / 42 / 41, 64 (402M) 72 / 48 / 60
//   128 of 512 x 2048 top 1 (a CTA of the down launch has one routed expert): 41 tokens (144M) 66 / 55 / 52, 64 (241M) 83 / 60 / 73
// and on layers that pairs.cu does not take, list / tiles: 8 of 2880 x 1024 top 2: 8 tokens (79M) 42 / 52, 12 (145M) 51 / 55, 16 (215M) 59 / 56
constexpr int kPairTokens = 64;
constexpr double kPairAgain = 170e6, kPairAgainFew = 275e6;   // ... and with at least four experts per token, up to 40 tokens
double weights_again(const chimere_moe_layer* w, int T) {
    const double distinct = w->E * (1.0 - std::pow(1.0 - (double)w->top_k / w->E, T));
    return (w->act == CHIMERE_ACT_SWIGLU ? 3.0 : 2.0) * w->H * (((double)T * w->top_k - distinct) * w->F + (T - 1.0) * w->F_s);
}
// (w here and below: without a K-quant shared expert)
bool few_per_expert(const chimere_moe_layer* w, int T) {
    const int64_t P = (int64_t)T * w->top_k;
    return T <= 4 || (T <= 40 && ((int64_t)w->F * w->H > (1 << 21) ? 16 * P <= 9 * w->E : 4 * P <= 5 * w->E));
}
bool pair_batch(const chimere_moe_layer* w, int T) {
    return few_per_expert(w, T) || (T <= kPairTokens && weights_again(w, T) <= (w->top_k >= 4 && T <= kFewTokens ? kPairAgainFew : kPairAgain));
}
bool list_batch(const chimere_moe_layer* w, int T) { return T <= kFewTokens && (few_per_expert(w, T) || weights_again(w, T) <= kPairAgain); }
// Upwards the tiles, which fetch and decode an expert's weights again for every 16 pairs, end where the grouped GEMM (64 pairs at a time) is the faster:
// a number of weights times pairs, less of them for wide rows, whose experts do not stay in L2 from one tile to the next, and for IQ3_S, whose sub-block
// factors are unpacked along.  us per layer, tiles / GEMM:
//   256 Q4_0 experts of 512 x 2048, top 8, 6144 tokens (52G) 2462 / 2514, 8192 (69G) 3704 / 3291; IQ3_S, 1024 tokens (9G) 521 / 598, 3072 (26G) 1367 / 1381,
//   4096 (34G) 1776 / 1730, and 64 of them, 1024 (9G) 1.03 times faster, 2048 (17G) 0.99
//   128 of 1024 x 2048, 768 tokens (13G) 1.01, 1024 (17G) 0.99; 64 of 1408 x 2048, top 6, 1024 (18G) 748 / 770; 128 of 1856 x 2688, 512 (15G) 703 / 731, 1024 (31G) 1240 / 1206, skewed 632 / 624 and 1194 / 1121
//   64 of 1536 x 4096, 256 tokens (13G) 683 / 687, 512 (26G) 1192 / 971; 8 of them, 512 (6G) 1.07, 768 (10G) 0.93; IQ3_S, 32 of them, 256 (6G) 1.03, 384 (10G) 0.93
//   (of 1024 x 1024 and smaller the tiles are the faster at any size that was tried, IQ3_S 256 x 1024 up to 4096 tokens, 9G: 1.00)
bool tile_batch(const chimere_moe_layer* w, int T) {
    const bool iq3 = w->type_up == CHIMERE_TYPE_IQ3_S;
    const double most = w->H <= 1024 ? (iq3 ? 8e9 : 64e9) : w->H <= 2048 && w->F <= 768 ? (iq3 ? 12e9 : 54e9) : w->H <= 2816 ? (iq3 ? 8e9 : 18e9) : iq3 ? 5e9 : 10e9;
    return (double)T * w->top_k * w->F * w->H <= most;
}
// ... and in the prefill entry: the tiles up to five pairs per expert, then the tcgen05 GEMM (GEMM / tiles: 256 experts 128 tokens 254 / 175 us,
// 256: 278 / 219, 777: 378 / 425, skewed 128: 109 / 102, 256: 144 / 156; 128 of 1856 x 2688 128 tokens 331 / 298, 256: 374 / 437).
// Of wide experts the two sides part below that line already, by the routing, which the host does not know: 128 of 1856 x 2688, 66 tokens 308 / 254 uniform and
// 138 / 133 skewed, 106: 326 / 285 and 160 / 185; 128 of 1536 x 4096, 80: 506 / 431 and 242 / 277; 128 of 2048 x 2048 top 4, 64: 306 / 240 and 103 / 98,
// 160: 378 / 312 and 157 / 185; 64 of 4096 x 1024, 24: 205 / 169 and 92 / 109.  The line stands for the even routing that such layers are trained to.  (Both launched,
// and a count of the tiles beyond an expert's first in each one's prologue to say which has work: skewed batches within 5 % of the better side, even ones 9 to
// 14 us slower for the launches that find nothing to do.)
bool prefill_mma(const chimere_moe_layer* w, int T) { return (int64_t)T * w->top_k <= 5 * (int64_t)w->E; }

// Layers that neither takes (experts and shared expert of different packed types, rows too long for the tiles' shared memory), and batches above tile_batch():
// From forward_gemm_tokens() tokens on the decode entry sends experts with at least kForwardGemmPairs pairs, and the shared expert,
// to the grouped GEMM and the others to the GEMV kernels: a GEMM tile costs the same with 1 pair as with 16, a GEMV entry grows
// with every pair.  Q4_0, us per layer, GEMV kernels alone / with the GEMM, uniform and (skewed) routing:
//   256 experts of  512 x 2048: 32 tokens  95 / 127 (86 / 85),   40: 114 / 148 (103 / 99),  41: 168 / 151 (120 / 99)
//   128 of 768 x 2048:          40 tokens 158 / 175,  41: 200 / 177;     128 of 1024 x 2048: 24: 152 / 149 (148 / 91),  40: 208 / 204 (194 / 116)
//   64 of 1408 x 2048:          17 tokens 132 / 142,  24: 168 / 169;     128 of 1856 x 2688:  9: 111 / 118 (97 / 93),   17: 180 / 170 (164 / 122)
// (From 41 tokens on the GEMV entries carry up to eight pairs.)  The best line depends on the routing, which the host does not know: at 17
// and 41 uniform routing loses 8 % at most and skewed routing gains.  Between 1024 and 1408 columns nothing was measured.
constexpr int kForwardGemmPairs = 3;
int forward_gemm_tokens(const chimere_moe_layer* w) { return (int64_t)w->F * w->H > (1 << 21) ? 17 : 41; }
static_assert(kForwardGemmPairs <= kMaxGroupTokens + 1, "a small expert must fit one work entry");
// ---------------------------------------------------------------- grouped GEMM path ----
// Token tiles of a batch: at most P / widest full ones and one partial one per expert with pairs, and the shared expert's.
constexpr int kTileColumns = 128, kForwardTileColumns = 64;   // columns of a full token tile: prefill / decode entry
int n_tiles_max_for(const chimere_moe_layer* w, int T, int widest) {
    const int P = T * w->top_k;
    return P / widest + (w->E < P ? w->E : P) + (w->F_s > 0 ? kshared(w) ? (T + 31) / 32 : (T + widest - 1) / widest : 0);
}
// ... and their columns / 16: a tile of n pairs is at most max(16, 2 n) columns wide.
int64_t n_col16_max_for(const chimere_moe_layer* w, int T) {
    const int64_t P = (int64_t)T * w->top_k, E = w->E < P ? w->E : P;
    const int64_t sh = w->F_s > 0 ? T : 0;
    return (2 * (P + sh) + 15) / 16 + E + 1;
}
int prefill_dims_ok(const chimere_moe_layer* w) {
    const int rpt = w->act == CHIMERE_ACT_SWIGLU ? 64 : 32;
    if (w->H % 128 || w->F % rpt || w->F_s % rpt) return 0;
    return 1;
}
struct PrefillArena { size_t tiles, bx, b2, sh_rows, total; int64_t bx_col16, b2_col16; };
PrefillArena prefill_arena(const chimere_moe_layer* w, int T) {
    PrefillArena A{};
    const int Fmax = w->F > w->F_s ? w->F : w->F_s;
    const int per = kshared_gemm(w) ? 640 : 576;   // 16 columns: 36 bytes per column and block, 40 with the blocks' sums
    A.bx_col16 = (int64_t)(w->H / 32) * per;
    A.b2_col16 = (int64_t)(Fmax / 32) * per;
    const int64_t cols = n_col16_max_for(w, T);
    size_t o = 0;
    A.tiles = o; o += up256((size_t)(8 + 4 * n_tiles_max_for(w, T, kForwardTileColumns)) * 4);
    A.bx = o; o += up256((size_t)(cols * A.bx_col16));
    A.b2 = o; o += up256((size_t)(cols * A.b2_col16));
    // a K-quant shared expert's output rows: the workspace's per-pair rows have no room for them (its layout is that of the
    // routed experts alone, so that layers with other shared experts can use the same workspace)
    A.sh_rows = o; o += kshared_gemm(w) ? up256((size_t)T * w->H * 4) : 0;
    A.total = o;
    return A;
}
// Whether the decode entry may take the grouped GEMM for T tokens of a layer (w without a K-quant shared expert): weights it
// reads in the tiled32 form, and enough tokens.
bool packed_types(const chimere_moe_layer* w) {
    auto ok = [](int t) { return t == CHIMERE_TYPE_Q4_0 || t == CHIMERE_TYPE_IQ3_S; };
    return ok(w->type_up) && ok(w->type_down) && (w->F_s == 0 || (ok(w->type_sh_up) && ok(w->type_sh_down)));
}
bool forward_gemm(const chimere_moe_layer* w, int T) {
    return T >= forward_gemm_tokens(w) && w->layout == CHIMERE_LAYOUT_TILED32 && prefill_dims_ok(w) && packed_types(w);
}
// Whether a batch is too small for the prefill entry's GEMM: tiles of mostly one pair.  256 IQ3_S experts of 512 x 2048, 16 tokens: uniform
// routing 115 us on the GEMM, 57 as decode, 48 on the pair kernels (103 when the prefill entry left experts of fewer than eight pairs to the GEMV kernels), skewed
// routing 47 and 53; eight experts, one token 43 and 26.  Q8_0 weights, whose GEMV entries fill an SM each, are the faster on the GEMM at one token.
bool prefill_as_decode(const chimere_moe_layer* w, int T) { return 2 * (int64_t)T * w->top_k <= w->E && packed_types(w); }

struct Layout {
    size_t topk_idx, topk_w, logits, sh_logit, x_q8, perm, offsets, group_list, counters, inter_q8, pair_out, status, total;
    size_t x_q, x_d, inter_q, inter_d;
    int x_d_stride, inter_d_stride, Fmax;
    int max_entries, n_row_tiles, tile_rows, n_counters;
    int n_row_tiles_tiled;
    size_t inter_stride;
    size_t gemm, gemm_bytes;   // the decode entry's token tiles (gemm_bytes = 0: never on the GEMM)
};

int entries_for(const chimere_moe_layer* w, int T, int group) {
    const int P = T * w->top_k, routed = (w->E < P ? w->E : P) + P / group;
    return (routed < P ? routed : P) + (w->F_s > 0 ? (T + shared_group_tokens(T) - 1) / shared_group_tokens(T) : 0);
}
bool wide_weights(const chimere_moe_layer* w) {
    return w->layout == CHIMERE_LAYOUT_GGML || w->type_up == CHIMERE_TYPE_Q8_0 || w->type_down == CHIMERE_TYPE_Q8_0;
}
int layer_group(const chimere_moe_layer* w, int T) { return group_tokens(T, (int64_t)w->F * w->H, wide_weights(w)); }
int max_entries_for(const chimere_moe_layer* w, int T) { return entries_for(w, T, layer_group(w, T)); }
// Entries that any batch of up to T tokens may need: between two steps of the entries' size their number grows with the batch, so the
// last batch before each step and T itself decide.  (The shortest entries: layers of different widths and types may share a workspace.)
int list_capacity(const chimere_moe_layer* w, int T) {
    int most = entries_for(w, T, group_tokens(T, 0, false));
    for (int t : kEntrySteps)
        if (t < T && entries_for(w, t, group_tokens(t, 0, false)) > most) most = entries_for(w, t, group_tokens(t, 0, false));
    return most;
}

Layout make_layout(const chimere_moe_layer* w, int T) {
    if (kshared(w)) { const chimere_moe_layer r = routed_only(w); return make_layout(&r, T); }
    Layout L{};
    const int k = w->top_k, H = w->H, E = w->E;
    const int Fmax = w->F > w->F_s ? w->F : w->F_s;
    const size_t pairs = (size_t)T * k + (w->F_s > 0 ? T : 0);
    L.max_entries = list_capacity(w, T);
    L.tile_rows = down_tile_rows(w->type_down, w->F, w->type_sh_down, w->F_s);
    L.n_row_tiles = (H + L.tile_rows - 1) / L.tile_rows;
    L.n_row_tiles_tiled = (H + 31) / 32;   // counters for the finest row tiling any batch size may choose
    const int max_tiles = L.n_row_tiles > L.n_row_tiles_tiled ? L.n_row_tiles : L.n_row_tiles_tiled;
    L.n_counters = kCtrRouteTile + (T + 7) / 8 + T * max_tiles;
    L.inter_stride = ((size_t)(Fmax / 32) * kQ81Bytes + 15) & ~(size_t)15;   // rows start on 16-byte boundaries (bulk copies)
    size_t o = 0;
    L.topk_idx = o; o += up256((size_t)T * k * 4);
    L.topk_w = o; o += up256((size_t)T * k * 4);
    L.logits = o; o += up256((size_t)T * E * 4);
    L.sh_logit = o; o += up256((size_t)T * 4);
    L.x_q8 = o; o += up256((size_t)T * (H / 32) * kQ81Bytes);
    L.perm = o; o += up256((size_t)T * k * 4);
    L.offsets = o; o += up256((size_t)(E + 1) * 4);
    L.group_list = o; o += up256((size_t)(kListHeader + kListEntry * L.max_entries) * 4);
    L.counters = o; o += up256((size_t)L.n_counters * 4);
    L.inter_q8 = o; o += up256(pairs * L.inter_stride);
    L.Fmax = Fmax;
    L.x_d_stride = (H / 32 + 3) & ~3;
    L.inter_d_stride = (Fmax / 32 + 3) & ~3;
    L.x_q = o; o += up256((size_t)T * H);
    L.x_d = o; o += up256((size_t)T * L.x_d_stride * 4);
    L.inter_q = o; o += up256(pairs * Fmax);
    L.inter_d = o; o += up256(pairs * L.inter_d_stride * 4);
    L.status = o; o += 256;
    L.pair_out = o; o += up256(pairs * H * 4);
    L.gemm = o;
    L.gemm_bytes = forward_gemm(w, T) ? prefill_arena(w, T).total : 0;
    o += up256(L.gemm_bytes);
    L.total = o;
    return L;
}

int cuda_rc(cudaError_t e) { return e == cudaSuccess ? 0 : -100 - (int)e; }

}  // namespace

extern "C" {

int chimere_b200_abi_version(void) { return 1; }
int chimere_b200_built_for_sm(void) { return 100; }

size_t chimere_b200_moe_workspace_bytes(const chimere_moe_layer* w, int max_T) {
    if (validate_layer(w) != 0 || max_T <= 0) return 0;
    return make_layout(w, max_T).total;
}

int chimere_b200_moe_workspace_init(chimere_moe_workspace* ws, void* d_arena, size_t bytes, const chimere_moe_layer* w,
                                    int max_T, cudaStream_t stream) {
    if (!ws || !d_arena) return -1;
    int rc = validate_layer(w);
    if (rc) return rc;
    if (max_T <= 0) return -2;
    if ((uintptr_t)d_arena & 255) return -5;
    const Layout L = make_layout(w, max_T);
    if (bytes < L.total) return -4;
    uint8_t* base = (uint8_t*)d_arena;
    std::memset(ws, 0, sizeof(*ws));
    ws->max_T = max_T;
    ws->topk_idx = (int32_t*)(base + L.topk_idx);
    ws->topk_w = (float*)(base + L.topk_w);
    ws->router_logits = (float*)(base + L.logits);
    ws->sh_gate_logit = (float*)(base + L.sh_logit);
    ws->x_q8 = base + L.x_q8;
    ws->perm = (int32_t*)(base + L.perm);
    ws->offsets = (int32_t*)(base + L.offsets);
    ws->group_list = (int32_t*)(base + L.group_list);
    ws->counters = (int32_t*)(base + L.counters);
    ws->inter_q8 = base + L.inter_q8;
    ws->pair_out = (float*)(base + L.pair_out);
    ws->x_q = (int8_t*)(base + L.x_q);
    ws->x_d = (float*)(base + L.x_d);
    ws->inter_q = (int8_t*)(base + L.inter_q);
    ws->inter_d = (float*)(base + L.inter_d);
    ws->status = (int32_t*)(base + L.status);
    if (L.gemm_bytes) { ws->prefill_arena = base + L.gemm; ws->prefill_bytes = L.gemm_bytes; }
    cudaError_t e = cudaMemsetAsync(ws->counters, 0, (size_t)L.n_counters * 4, stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(ws->status, 0, 256, stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(ws->group_list, 0, (size_t)(kListHeader + kListEntry * L.max_entries) * 4, stream);
    return cuda_rc(e);
}

static RouteParams route_params(const chimere_moe_layer* w, const float* d_x, int T, chimere_moe_workspace* ws, bool keep_gate_vector = false) {
    RouteParams p{};
    p.T = T; p.H = w->H; p.E = w->E; p.top_k = w->top_k; p.route_mode = w->route_mode;
    p.has_shared = w->F_s > 0;
    p.route_scale = w->route_scale;
    p.group = layer_group(w, T);
    p.x = d_x; p.router_w = w->router_w; p.router_bias = w->router_bias;
    p.shexp_gate_w = (w->F_s > 0 || keep_gate_vector) ? w->shexp_gate_w : nullptr;
    p.router_logits = ws->router_logits; p.sh_gate_logit = ws->sh_gate_logit;
    p.topk_idx = ws->topk_idx; p.topk_w = ws->topk_w; p.x_q8 = ws->x_q8;
    p.perm = ws->perm; p.offsets = ws->offsets; p.group_list = ws->group_list; p.counters = ws->counters;
    p.x_soa_q = ws->x_q; p.x_soa_d = ws->x_d; p.x_soa_d_stride = (w->H / 32 + 3) & ~3;
    p.status = ws->status;
    // the dispatch of a large batch counts in the memory of the down stage's combine counters (zero between the stages'
    // uses, and large enough from a few dozen tokens on)
    const Layout L = make_layout(w, ws->max_T);
    p.list_capacity = L.max_entries;
    const size_t combine_ints = (size_t)L.n_counters - kCtrRouteTile - (ws->max_T + 7) / 8;
    const size_t need = dispatch_scratch_ints(T, w->top_k);
    // the router of a large batch rewrites its rows into the per-pair output area, which the down stage fills only later; its
    // first T rows may hold the input (the residual + norm entry)
    p.scratch = ws->pair_out + (size_t)T * w->H;
    p.scratch_floats = ((size_t)ws->max_T * (w->top_k + (w->F_s > 0 ? 1 : 0)) - T) * w->H;
    p.dispatch_scratch = need <= combine_ints ? ws->counters + kCtrRouteTile + (ws->max_T + 7) / 8 : nullptr;
    return p;
}

static int check_call(const chimere_moe_layer* w, const void* a, const void* b, int T, const chimere_moe_workspace* ws,
                      bool allow_kquant_shared = false) {
    int rc = validate_layer(w);
    if (rc) return rc;
    if (kshared(w) && !allow_kquant_shared) return -6;   // only the whole-layer entries take a K-quant shared expert
    if (!a || !b || !ws || !ws->counters) return -1;
    if (T <= 0 || T > ws->max_T) return -2;
    return 0;
}

int chimere_b200_moe_route(const chimere_moe_layer* w, const float* d_x, int T, chimere_moe_workspace* ws,
                           cudaStream_t stream) {
    int rc = check_call(w, d_x, d_x, T, ws);
    if (rc) return rc;
    return cuda_rc(launch_route(route_params(w, d_x, T, ws), stream));
}

static int kshared_chain(const chimere_moe_layer* w, int T, float* d_y, chimere_moe_workspace* ws, cudaStream_t stream);
static int gemm_experts(const chimere_moe_layer* w, const chimere_moe_prefill_weights* pw, int E, int T, chimere_moe_workspace* ws, cudaStream_t stream,
                        const void* d_packed = nullptr, int row_bytes = 0, bool mixed = false, bool mma = false);
static cudaError_t finish_tokens(const chimere_moe_layer* w, float* d_y, int T, chimere_moe_workspace* ws, cudaStream_t stream);
static float* gemm_shared_rows(const chimere_moe_layer* w, int T, const chimere_moe_workspace* ws);
static GemvParams gate_up_params(const chimere_moe_layer* w, int T, chimere_moe_workspace* ws, const Layout& L);
static GemvParams down_params(const chimere_moe_layer* w, float* d_y, int T, chimere_moe_workspace* ws, const Layout& L);

int chimere_b200_moe_permute(const chimere_moe_layer* w, int T, chimere_moe_workspace* ws, cudaStream_t stream) {
    // The routing launch already leaves perm / offsets / the work list behind; this entry is for callers
    // that write ws->topk_idx themselves.  It runs only the dispatch step (no shared-expert entries).
    int rc = check_call(w, ws, ws, T, ws);
    if (rc) return rc;
    RouteParams p = route_params(w, nullptr, T, ws);
    p.has_shared = 0;
    return cuda_rc(launch_permute(p, stream));
}

// ---------------------------------------------------------------- expert-parallel pieces ----
int chimere_b200_moe_route_home(const chimere_moe_layer* w, const float* d_x, int T, chimere_moe_workspace* ws,
                                cudaStream_t stream) {
    int rc = check_call(w, d_x, d_x, T, ws);
    if (rc) return rc;
    RouteParams p = route_params(w, d_x, T, ws);
    p.list_mode = 1;   // work list: shared-expert entries only; the routed pairs go to their owners
    return cuda_rc(launch_route(p, stream));
}

int chimere_b200_moe_shared_expert(const chimere_moe_layer* w, int T, chimere_moe_workspace* ws, cudaStream_t stream) {
    int rc = check_call(w, ws, ws, T, ws);
    if (rc) return rc;
    if (w->layout != CHIMERE_LAYOUT_TILED32) return -2;
    if (w->F_s <= 0) return 0;
    const Layout L = make_layout(w, ws->max_T);
    const int max_entries = (T + shared_group_tokens(T) - 1) / shared_group_tokens(T);   // the home rank's list holds nothing else
    cudaError_t e = launch_gate_up_tiled(gate_up_params(w, T, ws, L), max_entries, stream);
    if (e != cudaSuccess) return cuda_rc(e);
    GemvParams g = down_params(w, nullptr, T, ws, L);
    g.no_combine = 1;
    return cuda_rc(launch_down_tiled(g, max_entries, stream));
}

static int run_experts(const chimere_moe_layer* w_local, int n_rows, const void* d_packed, int row_bytes, chimere_moe_workspace* ws,
                       cudaStream_t stream, int32_t* wait_flags = nullptr, int wait_n = 0, int wait_expect = 0) {
    if (n_rows == 0) return 0;
    int rc = check_call(w_local, ws, ws, n_rows, ws);
    if (rc) return rc;
    if (w_local->layout != CHIMERE_LAYOUT_TILED32 || w_local->top_k != 1 || w_local->F_s != 0) return -2;
    const int ds = (w_local->H / 32 + 3) & ~3;
    if (d_packed && (row_bytes % 16 || row_bytes < w_local->H + 4 * ds + 4)) return -2;
    RouteParams p = route_params(w_local, nullptr, n_rows, ws);
    p.has_shared = 0;
    if (d_packed) {   // ids sit behind the planes of every packed row
        p.topk_idx = (int32_t*)((uint8_t*)d_packed + w_local->H + 4 * ds);
        p.idx_stride = row_bytes / 4;
    }
    p.wait_flags = wait_flags; p.wait_n = wait_n; p.wait_expect = wait_expect;
    cudaError_t e = launch_permute(p, stream);
    if (e != cudaSuccess) return cuda_rc(e);
    const Layout L = make_layout(w_local, ws->max_T);
    const int max_entries = max_entries_for(w_local, n_rows);
    GemvParams gu = gate_up_params(w_local, n_rows, ws, L);
    if (d_packed) {
        gu.in_soa_q = (const int8_t*)d_packed; gu.in_soa_q_stride = row_bytes;
        gu.in_soa_d = (const float*)((const uint8_t*)d_packed + w_local->H); gu.in_soa_d_stride = row_bytes / 4;
        gu.few_tokens = 1;   // a fixed-size exchange: most of the n_rows slots carry no pair
    }
    e = launch_gate_up_tiled(gu, max_entries, stream);
    if (e != cudaSuccess) return cuda_rc(e);
    GemvParams g = down_params(w_local, nullptr, n_rows, ws, L);
    g.no_combine = 1;
    g.few_tokens = d_packed ? 1 : 0;
    return cuda_rc(launch_down_tiled(g, max_entries, stream));
}

int chimere_b200_moe_experts(const chimere_moe_layer* w_local, int n_rows, chimere_moe_workspace* ws, cudaStream_t stream) {
    return run_experts(w_local, n_rows, nullptr, 0, ws, stream);
}

int chimere_b200_moe_experts_packed(const chimere_moe_layer* w_local, int n_rows, const void* d_rows, int row_bytes,
                                    chimere_moe_workspace* ws, cudaStream_t stream) {
    if (n_rows == 0) return 0;
    if (!d_rows) return -1;
    return run_experts(w_local, n_rows, d_rows, row_bytes, ws, stream);
}

int chimere_b200_moe_experts_packed_p2p(const chimere_moe_layer* w_local, int n_rows, const void* d_rows, int row_bytes, int32_t* d_flags,
                                        int world, int cap, chimere_moe_workspace* ws, cudaStream_t stream) {
    if (!d_rows || !d_flags) return -1;
    if (world <= 0 || world > 32 || cap <= 0) return -2;
    return run_experts(w_local, n_rows, d_rows, row_bytes, ws, stream, d_flags, world, cap);
}

int chimere_b200_moe_ep_pack(const chimere_moe_layer* w, int T, chimere_moe_workspace* ws, void* d_send, int32_t* d_slot,
                             int experts_per_rank, int world, int cap, int row_bytes, cudaStream_t stream) {
    int rc = check_call(w, d_send, d_slot, T, ws);
    if (rc) return rc;
    const int ds = (w->H / 32 + 3) & ~3;
    if (experts_per_rank <= 0 || world <= 0 || world * experts_per_rank != w->E || cap < T * w->top_k) return -2;
    if (row_bytes % 16 || row_bytes < w->H + 4 * ds + 4 || w->H % 16) return -2;
    return cuda_rc(launch_ep_pack(ws->topk_idx, ws->x_q, ws->x_d, ds, (uint8_t*)d_send, d_slot, T, w->top_k, w->H, experts_per_rank,
                                  world, cap, row_bytes, stream));
}

int chimere_b200_moe_ep_finish(const chimere_moe_layer* w, const float* d_rows, const int32_t* d_slot, int T,
                               chimere_moe_workspace* ws, float* d_y, cudaStream_t stream) {
    int rc = check_call(w, d_rows, d_y, T, ws);
    if (rc) return rc;
    const float* shared_rows = w->F_s > 0 ? ws->pair_out + (size_t)T * w->top_k * w->H : nullptr;
    const float* logit = (w->F_s > 0 && w->shexp_gate_w) ? ws->sh_gate_logit : nullptr;
    return cuda_rc(launch_ep_finish(d_rows, d_slot, ws->topk_w, shared_rows, logit, d_y, T, w->H, w->top_k, stream));
}

// ---- exchange by peer stores (decode-size batches) ----
int chimere_b200_moe_ep_pack_p2p(const chimere_moe_layer* w, int T, chimere_moe_workspace* ws, void* const* d_peer_recv,
                                 int32_t* const* d_peer_flags, int32_t* d_ctr, int rank, int experts_per_rank, int world, int cap,
                                 int row_bytes, cudaStream_t stream) {
    int rc = check_call(w, d_peer_recv, d_peer_flags, T, ws);
    if (rc) return rc;
    if (!d_ctr) return -1;
    const int ds = (w->H / 32 + 3) & ~3;
    if (experts_per_rank <= 0 || world <= 0 || world * experts_per_rank != w->E || cap < T * w->top_k || rank < 0 || rank >= world) return -2;
    if (row_bytes % 16 || row_bytes < w->H + 4 * ds + 12 || w->H % 16) return -2;
    (void)d_ctr;
    return cuda_rc(launch_ep_pack_p2p(ws->topk_idx, ws->topk_w, ws->x_q, ws->x_d, ds, (uint8_t* const*)d_peer_recv, d_peer_flags, rank, T,
                                      w->top_k, w->H, experts_per_rank, world, cap, row_bytes, stream));
}

int chimere_b200_moe_ep_wait(int32_t* d_flags, int world, int cap, chimere_moe_workspace* ws, cudaStream_t stream) {
    if (!d_flags || !ws) return -1;
    if (world <= 0 || world > 32 || cap <= 0) return -2;
    return cuda_rc(launch_ep_wait_flags(d_flags, world, cap, ws->status, stream));
}

int chimere_b200_moe_ep_return_p2p(const chimere_moe_layer* w_local, chimere_moe_workspace* ws_owner, const void* d_rows, int row_bytes,
                                   float* const* d_peer_back, int32_t* const* d_peer_flags, int32_t* d_ctr, int rank, int world, int T, int cap,
                                   cudaStream_t stream) {
    if (!w_local || !ws_owner || !ws_owner->pair_out || !d_rows || !d_peer_back || !d_peer_flags || !d_ctr) return -1;
    const int ds = (w_local->H / 32 + 3) & ~3;
    if (world <= 0 || rank < 0 || rank >= world || T <= 0 || cap <= 0 || world * cap > ws_owner->max_T) return -2;
    if (row_bytes % 16 || row_bytes < w_local->H + 4 * ds + 12) return -2;
    (void)d_ctr;
    return cuda_rc(launch_ep_return_p2p(ws_owner->pair_out, (const uint8_t*)d_rows, row_bytes, w_local->H + 4 * ds, d_peer_back, d_peer_flags,
                                        rank, world, T, cap, w_local->H, stream));
}

int chimere_b200_moe_ep_finish_p2p(const chimere_moe_layer* w, const float* d_back, int32_t* d_flags, int world, int T,
                                   chimere_moe_workspace* ws, float* d_y, int32_t* d_ctr, cudaStream_t stream) {
    int rc = check_call(w, d_back, d_y, T, ws);
    if (rc) return rc;
    if (!d_flags || !d_ctr) return -1;
    if (world <= 0 || world > 32) return -2;
    const float* shared_rows = w->F_s > 0 ? ws->pair_out + (size_t)T * w->top_k * w->H : nullptr;
    const float* logit = (w->F_s > 0 && w->shexp_gate_w) ? ws->sh_gate_logit : nullptr;
    return cuda_rc(launch_ep_finish_p2p(d_back, d_flags, world, shared_rows, logit, d_y, T, w->H, d_ctr, ws->status, stream));
}

static GemvParams gate_up_params(const chimere_moe_layer* w, int T, chimere_moe_workspace* ws, const Layout& L) {
    GemvParams g{};
    g.T = T; g.top_k = w->top_k; g.H = w->H;
    g.act = w->act;
    g.few_limit = wide_weights(w) ? kFewTokensWide : kFewTokens;
    g.group_list = ws->group_list; g.perm = ws->perm;
    g.status = ws->status;
    g.ncols_routed = w->H; g.ncols_shared = w->H;
    g.nrows_routed = w->F; g.nrows_shared = w->F_s;
    g.type_routed = w->type_up; g.type_shared = w->type_sh_up;
    g.w_a = (const uint8_t*)w->gate_exps; g.w_b = (const uint8_t*)w->up_exps;
    g.stride_a = w->stride_gate; g.stride_b = w->stride_up;
    g.sh_a = (const uint8_t*)w->sh_gate; g.sh_b = (const uint8_t*)w->sh_up;
    g.in_q8 = ws->x_q8; g.in_stride = (int64_t)(w->H / 32) * kQ81Bytes;
    g.inter_q8 = ws->inter_q8; g.inter_stride = (int64_t)L.inter_stride;
    g.in_soa_q = ws->x_q; g.in_soa_q_stride = w->H; g.in_soa_d = ws->x_d; g.in_soa_d_stride = L.x_d_stride;
    g.out_soa_q = ws->inter_q; g.out_soa_q_stride = L.Fmax; g.out_soa_d = ws->inter_d; g.out_soa_d_stride = L.inter_d_stride;
    return g;
}

static GemvParams down_params(const chimere_moe_layer* w, float* d_y, int T, chimere_moe_workspace* ws, const Layout& L) {
    GemvParams g{};
    g.T = T; g.top_k = w->top_k; g.H = w->H;
    g.act = w->act;
    g.few_limit = wide_weights(w) ? kFewTokensWide : kFewTokens;
    g.group_list = ws->group_list; g.perm = ws->perm;
    g.status = ws->status;
    g.ncols_routed = w->F; g.ncols_shared = w->F_s;
    g.nrows_routed = w->H; g.nrows_shared = w->F_s > 0 ? w->H : 0;
    g.type_routed = w->type_down; g.type_shared = w->type_sh_down;
    g.w_a = (const uint8_t*)w->down_exps; g.stride_a = w->stride_down;
    g.sh_a = (const uint8_t*)w->sh_down;
    g.in_q8 = ws->inter_q8; g.in_stride = (int64_t)L.inter_stride;
    g.in_soa_q = ws->inter_q; g.in_soa_q_stride = L.Fmax; g.in_soa_d = ws->inter_d; g.in_soa_d_stride = L.inter_d_stride;
    g.pair_out = ws->pair_out; g.topk_w = ws->topk_w;
    g.sh_gate_logit = (w->F_s > 0 && w->shexp_gate_w) ? ws->sh_gate_logit : nullptr;
    g.y = d_y;
    g.combine_ctr = ws->counters + kCtrRouteTile + (ws->max_T + 7) / 8;
    g.tile_rows = L.tile_rows;
    g.n_row_tiles = (w->layout == CHIMERE_LAYOUT_TILED32)
                        ? (w->H + 32 * tiled_down_geom(w->type_down, w->F, w->type_sh_down, w->F_s, T).wr - 1) /
                              (32 * tiled_down_geom(w->type_down, w->F, w->type_sh_down, w->F_s, T).wr)
                        : L.n_row_tiles;
    return g;
}

static cudaError_t run_gate_up(const chimere_moe_layer* w, const GemvParams& g, int max_entries, cudaStream_t stream) {
    return w->layout == CHIMERE_LAYOUT_TILED32 ? launch_gate_up_tiled(g, max_entries, stream) : launch_gate_up(g, max_entries, stream);
}
static cudaError_t run_down(const chimere_moe_layer* w, const GemvParams& g, int max_entries, cudaStream_t stream) {
    return w->layout == CHIMERE_LAYOUT_TILED32 ? launch_down_tiled(g, max_entries, stream) : launch_down(g, max_entries, stream);
}

// ---- tiled32 packing ----
struct PackPlan { size_t gate, up, down, sh_gate, sh_up, sh_down, total; int64_t sg, su, sd; };
static PackPlan pack_plan(const chimere_moe_layer* w) {
    PackPlan P{};
    const bool dual = w->act == CHIMERE_ACT_SWIGLU;
    size_t o = 0;
    P.su = tiled_matrix_bytes(w->type_up, w->F, w->H);
    P.sg = dual ? tiled_matrix_bytes(w->type_gate, w->F, w->H) : 0;
    P.sd = tiled_matrix_bytes(w->type_down, w->H, w->F);
    P.gate = o; o += up256((size_t)P.sg * w->E);
    P.up = o; o += up256((size_t)P.su * w->E);
    P.down = o; o += up256((size_t)P.sd * w->E);
    if (w->F_s > 0) {
        P.sh_gate = o; o += dual ? up256((size_t)tiled_matrix_bytes(w->type_sh_gate, w->F_s, w->H)) : 0;
        P.sh_up = o; o += up256((size_t)tiled_matrix_bytes(w->type_sh_up, w->F_s, w->H));
        P.sh_down = o; o += up256((size_t)tiled_matrix_bytes(w->type_sh_down, w->H, w->F_s));
    }
    P.total = o;
    return P;
}

size_t chimere_b200_moe_pack_bytes(const chimere_moe_layer* raw) {
    if (validate_layer(raw) != 0 || raw->layout != CHIMERE_LAYOUT_GGML) return 0;
    if (kshared(raw)) { const chimere_moe_layer r = routed_only(raw); return pack_plan(&r).total; }
    return pack_plan(raw).total;
}

int chimere_b200_moe_pack(const chimere_moe_layer* raw, void* d_arena, size_t bytes, chimere_moe_layer* packed,
                          cudaStream_t stream) {
    int rc = validate_layer(raw);
    if (rc) return rc;
    if (!d_arena || !packed) return -1;
    if (kshared(raw)) {   // the routed experts are re-tiled; the K-quant shared matrices stay where and as they are
        const chimere_moe_layer r = routed_only(raw);
        rc = chimere_b200_moe_pack(&r, d_arena, bytes, packed, stream);
        if (rc) return rc;
        packed->F_s = raw->F_s; packed->sh_gate = raw->sh_gate; packed->sh_up = raw->sh_up; packed->sh_down = raw->sh_down;
        packed->type_sh_gate = raw->type_sh_gate; packed->type_sh_up = raw->type_sh_up; packed->type_sh_down = raw->type_sh_down;
        return 0;
    }
    if (raw->layout != CHIMERE_LAYOUT_GGML) return -2;
    if ((uintptr_t)d_arena & 255) return -5;
    const PackPlan P = pack_plan(raw);
    if (bytes < P.total) return -4;
    const bool dual = raw->act == CHIMERE_ACT_SWIGLU;
    uint8_t* base = (uint8_t*)d_arena;
    *packed = *raw;
    packed->layout = CHIMERE_LAYOUT_TILED32;
    cudaError_t e = cudaSuccess;
    if (dual) {
        e = launch_pack(raw->type_gate, raw->gate_exps, base + P.gate, raw->E, raw->F, raw->H, raw->stride_gate, P.sg, stream);
        packed->gate_exps = base + P.gate; packed->stride_gate = P.sg;
    }
    if (e == cudaSuccess) e = launch_pack(raw->type_up, raw->up_exps, base + P.up, raw->E, raw->F, raw->H, raw->stride_up, P.su, stream);
    packed->up_exps = base + P.up; packed->stride_up = P.su;
    if (e == cudaSuccess) e = launch_pack(raw->type_down, raw->down_exps, base + P.down, raw->E, raw->H, raw->F, raw->stride_down, P.sd, stream);
    packed->down_exps = base + P.down; packed->stride_down = P.sd;
    if (raw->F_s > 0) {
        if (dual) {
            if (e == cudaSuccess) e = launch_pack(raw->type_sh_gate, raw->sh_gate, base + P.sh_gate, 1, raw->F_s, raw->H, 0, 0, stream);
            packed->sh_gate = base + P.sh_gate;
        }
        if (e == cudaSuccess) e = launch_pack(raw->type_sh_up, raw->sh_up, base + P.sh_up, 1, raw->F_s, raw->H, 0, 0, stream);
        packed->sh_up = base + P.sh_up;
        if (e == cudaSuccess) e = launch_pack(raw->type_sh_down, raw->sh_down, base + P.sh_down, 1, raw->H, raw->F_s, 0, 0, stream);
        packed->sh_down = base + P.sh_down;
    }
    return cuda_rc(e);
}

size_t chimere_b200_packed_matrix_bytes(int wtype, int nrows, int ncols) {
    if (!type_ok(wtype) || nrows <= 0 || nrows % 32 || ncols <= 0 || ncols % type_cols_multiple(wtype)) return 0;
    return (size_t)tiled_matrix_bytes(wtype, nrows, ncols);
}

int chimere_b200_pack_matrix(int wtype, const void* d_raw, void* d_out, int nrows, int ncols, cudaStream_t stream) {
    if (!d_raw || !d_out) return -1;
    if (!type_ok(wtype)) return -3;
    if (nrows <= 0 || nrows % 32 || ncols <= 0 || ncols % type_cols_multiple(wtype)) return -2;
    return cuda_rc(launch_pack(wtype, d_raw, d_out, 1, nrows, ncols, 0, 0, stream));
}

int chimere_b200_block_sumi_tiled(int wtype, const void* d_packed, const void* d_xq8, int32_t* d_sumi, int ncols, int nrows,
                                  cudaStream_t stream) {
    if (!d_packed || !d_xq8 || !d_sumi) return -1;
    if (!type_ok(wtype)) return -3;
    if (ncols <= 0 || nrows < 0 || nrows % 32 || ncols % type_cols_multiple(wtype)) return -2;
    return cuda_rc(launch_block_sumi_tiled(wtype, d_packed, d_xq8, d_sumi, ncols, nrows, stream));
}

int chimere_b200_moe_gate_up(const chimere_moe_layer* w, int T, chimere_moe_workspace* ws, cudaStream_t stream) {
    int rc = check_call(w, ws, ws, T, ws);
    if (rc) return rc;
    const Layout L = make_layout(w, ws->max_T);
    return cuda_rc(run_gate_up(w, gate_up_params(w, T, ws, L), max_entries_for(w, T), stream));
}

int chimere_b200_moe_down_combine(const chimere_moe_layer* w, float* d_y, int T, chimere_moe_workspace* ws,
                                  cudaStream_t stream) {
    int rc = check_call(w, d_y, d_y, T, ws);
    if (rc) return rc;
    const Layout L = make_layout(w, ws->max_T);
    return cuda_rc(run_down(w, down_params(w, d_y, T, ws, L), max_entries_for(w, T), stream));
}

// Decode batches up to pair_batch()'s line run without a work list where the pair kernels take the layer: the router's logits, then
// two launches that select their experts themselves.  A K-quant shared expert rides along or follows as kshared_chain.
// Up to five tokens it rides along: a row of it decodes its blocks for every token, and kshared_chain for eight at a time.  us per layer (256 IQ3_S /
// Q4_0 experts, Q5_K shared, in the pair launches / behind them): 1 token 18.3 / 20.3, 4: 28.2 / 29.4, 5: 33.9 / 34.3, 6: 37.1 / 35.9, 12: 59.9 / 54.1,
// 33: 143.8 / 107.7 (123.9 on the work list).
constexpr int kPairKquantTokens = 5;
static PairExtras pair_extras(const chimere_moe_layer* w, int T, chimere_moe_workspace* ws) {
    PairExtras x{};
    if (!kshared(w) || T > kPairKquantTokens || !pairs_take_kquant(*w)) return x;
    x.type = w->type_sh_up; x.type_down = w->type_sh_down; x.F_s = w->F_s;
    x.gate = (const uint8_t*)w->sh_gate; x.up = (const uint8_t*)w->sh_up; x.down = (const uint8_t*)w->sh_down;
    x.rows = ws->pair_out;
    x.logit = w->shexp_gate_w ? ws->sh_gate_logit : nullptr;
    return x;
}
static bool pairs_forward(const chimere_moe_layer* w, int T, chimere_moe_workspace* ws) {
    const chimere_moe_layer wr = kshared(w) ? routed_only(w) : *w;
    if (!pair_batch(&wr, T) || w->layout != CHIMERE_LAYOUT_TILED32) return false;
    const Layout L = make_layout(&wr, ws->max_T);
    return pairs_run(gate_up_params(&wr, T, ws, L), down_params(&wr, nullptr, T, ws, L), pair_extras(w, T, ws));
}
static int run_pairs(const chimere_moe_layer* w, const float* d_x, const float* d_hidden, float* d_residual, const float* d_norm_weight, float eps, float* d_y, int T,
                     chimere_moe_workspace* ws, cudaStream_t stream) {
    const bool ks = kshared(w);
    const chimere_moe_layer wr = ks ? routed_only(w) : *w;
    const Layout L = make_layout(&wr, ws->max_T);
    PairExtras x = pair_extras(w, T, ws);
    RouteParams rp = route_params(&wr, d_x, T, ws, ks);
    rp.logits_only = 1;
    cudaError_t e;
    if (d_hidden) {
        x.hidden = d_hidden; x.residual = d_residual;
        e = launch_route_norm(rp, d_hidden, d_residual, d_norm_weight, eps, stream);
    } else e = launch_route(rp, stream);
    if (e == cudaSuccess) e = launch_pair_gate_up(rp, gate_up_params(&wr, T, ws, L), x, stream);
    if (e == cudaSuccess) e = launch_pair_down(rp, down_params(&wr, d_y, T, ws, L), x, stream);
    return e != cudaSuccess || !ks || x.type ? cuda_rc(e) : kshared_chain(w, T, d_y, ws, stream);
}

// Products of a batch on the warp-level MMA (mma_tiles.cu), 16 pairs of an expert at a time; w: without a K-quant shared expert.
static bool mma_runs(const chimere_moe_layer* w, int T, chimere_moe_workspace* ws) {
    if (w->layout != CHIMERE_LAYOUT_TILED32) return false;
    const Layout L = make_layout(w, ws->max_T);
    return mma_tiles_run(gate_up_params(w, T, ws, L), down_params(w, nullptr, T, ws, L));
}
static int run_mma(const chimere_moe_layer* w, int T, chimere_moe_workspace* ws, cudaStream_t stream) {
    const Layout L = make_layout(w, ws->max_T);
    cudaError_t e = launch_mma_gate_up(gate_up_params(w, T, ws, L), ws->offsets, w->E, stream);
    if (e == cudaSuccess) e = launch_mma_down(down_params(w, nullptr, T, ws, L), ws->offsets, w->E, stream);
    return cuda_rc(e);
}

int chimere_b200_moe_forward(const chimere_moe_layer* w, const float* d_x, float* d_y, int T, chimere_moe_workspace* ws,
                             cudaStream_t stream) {
    int rc = check_call(w, d_x, d_y, T, ws, true);
    if (rc) return rc;
    const bool ks = kshared(w);
    const chimere_moe_layer wr_ = ks ? routed_only(w) : *w;
    const chimere_moe_layer* wr = &wr_;
    cudaError_t e;
    const Layout L = make_layout(wr, ws->max_T);
    if (pairs_forward(w, T, ws)) return run_pairs(w, d_x, nullptr, nullptr, nullptr, 0.0f, d_y, T, ws, stream);
    const bool gemm = forward_gemm(wr, T) && ws->prefill_arena && ws->prefill_bytes >= prefill_arena(wr, ws->max_T).total &&
                      tiled_bulk_runs(gate_up_params(wr, T, ws, L), down_params(wr, d_y, T, ws, L));
    if (!list_batch(wr, T) && (tile_batch(wr, T) || !gemm) && mma_runs(wr, T, ws)) {
        RouteParams rp = route_params(wr, d_x, T, ws, ks);
        rp.list_mode = 2;
        e = launch_route(rp, stream);
        if (e != cudaSuccess) return cuda_rc(e);
        rc = run_mma(wr, T, ws, stream);
        if (rc) return rc;
        e = finish_tokens(wr, d_y, T, ws, stream);
    } else if (gemm) {
        RouteParams rp = route_params(wr, d_x, T, ws, ks);
        rp.list_mode = 2;
        e = launch_route(rp, stream);
        if (e != cudaSuccess) return cuda_rc(e);
        rc = gemm_experts(wr, nullptr, wr->E, T, ws, stream, nullptr, 0, true);
        if (rc) return rc;
        e = finish_tokens(wr, d_y, T, ws, stream);
    } else {
        const int max_entries = max_entries_for(wr, T);
        e = launch_route(route_params(wr, d_x, T, ws, ks), stream);
        if (e != cudaSuccess) return cuda_rc(e);
        e = run_gate_up(wr, gate_up_params(wr, T, ws, L), max_entries, stream);
        if (e != cudaSuccess) return cuda_rc(e);
        e = run_down(wr, down_params(wr, d_y, T, ws, L), max_entries, stream);
    }
    if (e != cudaSuccess || !ks) return cuda_rc(e);
    return kshared_chain(w, T, d_y, ws, stream);
}

// The device's address of `bytes` of pinned host memory; null for pageable memory and for ranges that the device does not see in one piece.  The
// kernels read and write such a range by themselves, so its end is looked at as well: memory that is pinned only up to somewhere inside the
// rows is refused, as a copy of it is.
static cudaError_t pinned_address(const float* h, size_t bytes, float** device) {
    const char* last = (const char*)h + bytes - 1;
    cudaPointerAttributes a{}, z{};
    *device = nullptr;
    const bool first_pinned = cudaPointerGetAttributes(&a, h) == cudaSuccess && a.type == cudaMemoryTypeHost && a.devicePointer;
    const bool last_pinned = first_pinned && cudaPointerGetAttributes(&z, last) == cudaSuccess && z.type == cudaMemoryTypeHost && z.devicePointer;
    if (!last_pinned) {
        (void)cudaGetLastError();   // (an unregistered pointer leaves an error behind on older runtimes)
        return first_pinned ? cudaErrorInvalidValue : cudaSuccess;
    }
    if ((const char*)z.devicePointer - (const char*)a.devicePointer == last - (const char*)h) *device = static_cast<float*>(a.devicePointer);
    return cudaSuccess;
}
constexpr size_t kFetchBytes = 256 * 1024;   // rows of up to so many bytes come in by a kernel

int chimere_b200_moe_forward_host(const chimere_moe_layer* w, const float* h_x, float* h_y, int T, float* d_x, float* d_y,
                                  chimere_moe_workspace* ws, cudaStream_t stream) {
    if (!h_x || !h_y) return -1;
    int rc = check_call(w, d_x, d_y, T, ws, true);
    if (rc) return rc;
    const size_t bytes = (size_t)T * w->H * sizeof(float);
    float *x_host = nullptr, *y_host = nullptr;
    cudaError_t e = bytes <= kFetchBytes ? pinned_address(h_x, bytes, &x_host) : cudaSuccess;
    if (e == cudaSuccess) e = x_host ? launch_fetch_rows(x_host, d_x, (int64_t)T * w->H, stream) : cudaMemcpyAsync(d_x, h_x, bytes, cudaMemcpyHostToDevice, stream);
    if (e != cudaSuccess) return cuda_rc(e);
    // A pinned result buffer is addressable from the device under a pointer of its own: the last kernel then stores y
    // straight into host memory and the copy back (a second trip through the copy engine, serial behind the kernels) is
    // not needed.  Pageable memory, or a K-quant shared expert as launches of its own (the last of which reads y back), takes the staged copy.
    // (Looked at while the rows are on their way.)
    if (!kshared(w) || (pairs_forward(w, T, ws) && pair_extras(w, T, ws).type)) e = pinned_address(h_y, bytes, &y_host);
    if (e != cudaSuccess) {
        (void)cudaStreamSynchronize(stream);   // (h_x is the caller's again)
        return cuda_rc(e);
    }
    float* y_dev = y_host ? y_host : d_y;
    rc = chimere_b200_moe_forward(w, d_x, y_dev, T, ws, stream);
    if (rc) return rc;
    if (y_dev == d_y) {
        e = cudaMemcpyAsync(h_y, d_y, bytes, cudaMemcpyDeviceToHost, stream);
        if (e != cudaSuccess) return cuda_rc(e);
    }
    return cuda_rc(cudaStreamSynchronize(stream));
}

int chimere_b200_block_sumi(int wtype, const void* d_w, const void* d_xq8, int32_t* d_sumi, int ncols, int nrows,
                            cudaStream_t stream) {
    if (!d_w || !d_xq8 || !d_sumi) return -1;
    if (!type_ok(wtype)) return -3;
    if (ncols <= 0 || nrows < 0 || ncols % type_cols_multiple(wtype)) return -2;
    return cuda_rc(launch_block_sumi(wtype, d_w, d_xq8, d_sumi, ncols, nrows, stream));
}

// ---------------------------------------------------------------- tcgen05 block-scaled GEMM --
size_t chimere_b200_mma128_bytes(int rows, int cols) {
    if (rows <= 0 || cols <= 0 || cols % 32) return 0;
    return (size_t)((rows + 127) / 128) * (cols / 32) * (4096 + 512);
}

int chimere_b200_pack_mma128(const int8_t* d_q, const float* d_scales, void* d_out, int rows, int cols, cudaStream_t stream) {
    if (!d_q || !d_scales || !d_out) return -1;
    if (rows <= 0 || cols <= 0 || cols % 32) return -2;
    return cuda_rc(launch_pack_mma128(d_q, d_scales, (uint8_t*)d_out, rows, cols, stream));
}

int chimere_b200_gemm_i8(const void* d_a, const void* d_b, int rows, int tokens, int cols, float* d_out, void* d_items,
                         int32_t* d_status, cudaStream_t stream) {
    if (!d_a || !d_b || !d_out || !d_items || !d_status) return -1;
    if (rows <= 0 || tokens <= 0 || cols <= 0 || cols % 32) return -2;
    const int rt = (rows + 127) / 128, tt = (tokens + 127) / 128, nb = cols / 32;
    std::vector<GemmItem> items;
    for (int i = 0; i < rt; ++i)
        for (int j = 0; j < tt; ++j) {
            GemmItem it{};
            it.a_offset = (int64_t)i * nb * (4096 + 512);
            it.b_offset = (int64_t)j * nb * (4096 + 512);
            it.n_valid = tokens - j * 128 < 128 ? tokens - j * 128 : 128;
            it.rows_valid = rows - i * 128 < 128 ? rows - i * 128 : 128;
            it.out_row0 = i * 128; it.out_col0 = j * 128;
            items.push_back(it);
        }
    cudaError_t e = cudaMemcpyAsync(d_items, items.data(), items.size() * sizeof(GemmItem), cudaMemcpyHostToDevice, stream);
    if (e != cudaSuccess) return cuda_rc(e);
    int32_t* counter = (int32_t*)((uint8_t*)d_items + items.size() * sizeof(GemmItem));   // the tile counter sits behind the list
    e = cudaMemsetAsync(counter, 0, 256, stream);
    if (e != cudaSuccess) return cuda_rc(e);
    e = cudaStreamSynchronize(stream);   // the host vector goes away; this entry is a test primitive, not the hot path
    if (e != cudaSuccess) return cuda_rc(e);
    GemmParams p{};
    p.a_base = (const uint8_t*)d_a; p.b_base = (const uint8_t*)d_b; p.items = (const GemmItem*)d_items; p.nblocks = nb;
    p.out = d_out; p.ldo = tokens; p.status = d_status;
    return cuda_rc(launch_gemm_i8_f32(p, (int)items.size(), counter, stream));
}

int chimere_b200_mma_i8_probe(int n_mma, int n_cols, int n_acc, int32_t* d_status, cudaStream_t stream) {
    if (n_mma <= 0 || n_mma % 64 || (n_cols != 128 && n_cols != 256) || n_acc < 1 || n_acc * n_cols > 512) return -2;
    return launch_mma_i8_probe(n_mma, n_cols, n_acc, d_status, stream);
}

// The GEMM reads 4-bit weights in the tiled32 form; Q8_0 matrices, and a shared expert in Q4_K / Q5_K super-blocks, get a copy
// in the MMA's own order (mma128 tiles; gate and up rows interleaved per 64, so that one output tile holds both).
namespace {
struct PrefillPlan { size_t gu, down, sh_gu, sh_down, total; int64_t sgu, sdown, s_sh_gu, s_sh_down; };
PrefillPlan prefill_plan(const chimere_moe_layer* w) {
    PrefillPlan P{};
    const int rpt = w->act == CHIMERE_ACT_SWIGLU ? 64 : 128;
    auto tiles = [](int rows, int per, int cols) { return (int64_t)((rows + per - 1) / per) * (cols / 32) * (4096 + 512); };
    P.sgu = w->type_up == CHIMERE_TYPE_Q8_0 ? tiles(w->F, rpt, w->H) : 0;
    P.sdown = w->type_down == CHIMERE_TYPE_Q8_0 ? tiles(w->H, 128, w->F) : 0;
    P.s_sh_gu = w->F_s > 0 && w->type_sh_up == CHIMERE_TYPE_Q8_0 ? tiles(w->F_s, rpt, w->H) : 0;
    P.s_sh_down = w->F_s > 0 && w->type_sh_down == CHIMERE_TYPE_Q8_0 ? tiles(w->H, 128, w->F_s) : 0;
    if (kshared_gemm(w)) {
        P.s_sh_gu = (int64_t)((w->F_s + 63) / 64) * (w->H / 128) * kOperandMinStage;
        P.s_sh_down = (int64_t)(w->H / 128) * (w->F_s / 128) * kOperandMinStage;
    }
    size_t o = 256;   // (never empty: the size doubles as the check of the dimensions)
    P.gu = o; o += up256((size_t)P.sgu * w->E);
    P.down = o; o += up256((size_t)P.sdown * w->E);
    P.sh_gu = o; o += up256((size_t)P.s_sh_gu);
    P.sh_down = o; o += up256((size_t)P.s_sh_down);
    P.total = o;
    return P;
}
}  // namespace

size_t chimere_b200_moe_pack_prefill_bytes(const chimere_moe_layer* raw) {
    if (validate_layer(raw) != 0) return 0;
    if (kshared(raw) && !kshared_gemm(raw)) { const chimere_moe_layer r = routed_only(raw); return chimere_b200_moe_pack_prefill_bytes(&r); }
    if (raw->layout != CHIMERE_LAYOUT_GGML || !prefill_dims_ok(raw)) return 0;
    return prefill_plan(raw).total;
}

int chimere_b200_moe_pack_prefill(const chimere_moe_layer* raw, void* d_arena, size_t bytes, chimere_moe_prefill_weights* out,
                                  cudaStream_t stream) {
    int rc = validate_layer(raw);
    if (rc) return rc;
    if (!d_arena || !out) return -1;
    if (kshared(raw) && !kshared_gemm(raw)) { const chimere_moe_layer r = routed_only(raw); return chimere_b200_moe_pack_prefill(&r, d_arena, bytes, out, stream); }
    if (raw->layout != CHIMERE_LAYOUT_GGML || !prefill_dims_ok(raw)) return -2;
    if ((uintptr_t)d_arena & 255) return -5;
    const PrefillPlan P = prefill_plan(raw);
    if (bytes < P.total) return -4;
    const bool dual = raw->act == CHIMERE_ACT_SWIGLU;
    uint8_t* base = (uint8_t*)d_arena;
    std::memset(out, 0, sizeof(*out));
    out->rows_per_gu_tile = dual ? 64 : 128;
    cudaError_t e = cudaSuccess;
    if (!dual && P.sgu + P.s_sh_gu > 0 && (raw->F % 128 || raw->F_s % 128)) e = cudaMemsetAsync(base, 0, P.total, stream);   // zero rows and scales behind the last real row
    auto gate_up = [&](const void* gate, const void* up, size_t at, int n, int rows, int64_t sg, int64_t su, int64_t so) {
        if (dual && e == cudaSuccess) e = launch_pack_mma128_q8_0(gate, base + at, n, rows, raw->H, 1, sg, so, stream);
        if (e == cudaSuccess) e = launch_pack_mma128_q8_0(up, base + at, n, rows, raw->H, dual ? 2 : 0, su, so, stream);
    };
    if (P.sgu) { gate_up(raw->gate_exps, raw->up_exps, P.gu, raw->E, raw->F, raw->stride_gate, raw->stride_up, P.sgu); out->gu_exps = base + P.gu; out->stride_gu = P.sgu; }
    if (P.sdown) {
        if (e == cudaSuccess) e = launch_pack_mma128_q8_0(raw->down_exps, base + P.down, raw->E, raw->H, raw->F, 0, raw->stride_down, P.sdown, stream);
        out->down_exps = base + P.down; out->stride_down = P.sdown;
    }
    if (kshared_gemm(raw)) {
        if (e == cudaSuccess) e = launch_pack_operand_min(raw->type_sh_gate, raw->sh_gate, base + P.sh_gu, raw->F_s, raw->H, 1, stream);
        if (e == cudaSuccess) e = launch_pack_operand_min(raw->type_sh_up, raw->sh_up, base + P.sh_gu, raw->F_s, raw->H, 2, stream);
        if (e == cudaSuccess) e = launch_pack_operand_min(raw->type_sh_down, raw->sh_down, base + P.sh_down, raw->H, raw->F_s, 0, stream);
        out->sh_gu = base + P.sh_gu; out->sh_down = base + P.sh_down;
        return cuda_rc(e);
    }
    if (P.s_sh_gu) { gate_up(raw->sh_gate, raw->sh_up, P.sh_gu, 1, raw->F_s, 0, 0, 0); out->sh_gu = base + P.sh_gu; }
    if (P.s_sh_down) {
        if (e == cudaSuccess) e = launch_pack_mma128_q8_0(raw->sh_down, base + P.sh_down, 1, raw->H, raw->F_s, 0, 0, 0, stream);
        out->sh_down = base + P.sh_down;
    }
    return cuda_rc(e);
}

size_t chimere_b200_moe_prefill_bytes(const chimere_moe_layer* w, int max_T) {
    if (validate_layer(w) != 0 || max_T <= 0) return 0;
    if (kshared(w) && !kshared_gemm(w)) { const chimere_moe_layer r = routed_only(w); return chimere_b200_moe_prefill_bytes(&r, max_T); }
    if (!prefill_dims_ok(w)) return 0;
    return prefill_arena(w, max_T).total;
}

// The K-quant shared expert of `w` for T tokens whose Q8_1 rows (ws->x_q8) and gate logits (ws->sh_gate_logit) the router
// left behind, added to d_y: up (and gate) GEMVs, activation + Q8_1, down GEMV with the sigmoid-gated add.  The f32 rows
// borrow ws->pair_out and the intermediates ws->inter_q8: the routed part of the call is done with both by then.
static int kshared_chain(const chimere_moe_layer* w, int T, float* d_y, chimere_moe_workspace* ws, cudaStream_t stream) {
    const bool dual = w->act == CHIMERE_ACT_SWIGLU;
    const int64_t x_stride = (int64_t)(w->H / 32) * kQ81Bytes, i_stride = (int64_t)(w->F_s / 32) * kQ81Bytes;
    float* up = ws->pair_out;
    float* gate = dual ? ws->pair_out + (size_t)T * w->F_s : nullptr;
    // gate and up share a launch when they have the same type; the three (or four) kernels are chained programmatically
    const bool one = dual && w->type_sh_gate == w->type_sh_up;
    cudaError_t e = launch_mmvq_kquant_batched(w->type_sh_up, w->sh_up, one ? w->sh_gate : nullptr, ws->x_q8, x_stride, up, one ? gate : nullptr,
                                               w->F_s, T, w->H, w->F_s, 0, nullptr, true, stream);
    if (e == cudaSuccess && dual && !one)
        e = launch_mmvq_kquant_batched(w->type_sh_gate, w->sh_gate, nullptr, ws->x_q8, x_stride, gate, nullptr, w->F_s, T, w->H, w->F_s, 0, nullptr,
                                       true, stream);
    if (e == cudaSuccess) e = launch_act_q8_1(gate, up, w->F_s, ws->inter_q8, i_stride, T, w->F_s, stream);
    if (e == cudaSuccess)
        e = launch_mmvq_kquant_batched(w->type_sh_down, w->sh_down, nullptr, ws->inter_q8, i_stride, d_y, nullptr, w->H, T, w->F_s, w->H,
                                       w->shexp_gate_w ? 2 : 1, w->shexp_gate_w ? ws->sh_gate_logit : nullptr, true, stream);
    return cuda_rc(e);
}

// One launch's view of the layer: where the matrices are and how they are cut into 128-row output tiles.
static PrefillGemmMats gemm_mats(const chimere_moe_layer* w, const chimere_moe_prefill_weights* pw, bool shared, bool down) {
    PrefillGemmMats m{};
    const bool dual = !down && w->act == CHIMERE_ACT_SWIGLU;
    const int width = shared ? w->F_s : w->F;
    const void* gate = shared ? w->sh_gate : w->gate_exps;
    const void* up = shared ? w->sh_up : w->up_exps;
    const void* dn = shared ? w->sh_down : w->down_exps;
    m.type = shared ? (down ? w->type_sh_down : w->type_sh_up) : (down ? w->type_down : w->type_up);
    m.ncols = down ? width : w->H;
    m.rows32 = (down ? w->H : width) / 32;
    m.row_tiles = dual ? (m.rows32 + 1) / 2 : (m.rows32 + 3) / 4;
    if (kquant_type(m.type)) {   // (a shared expert that kshared_gemm accepts: its copy with minimums)
        m.type = kTypeOperandMin;
        m.w0 = (const uint8_t*)(pw ? (down ? pw->sh_down : pw->sh_gu) : nullptr);
        return m;
    }
    m.tile_bytes = m.ncols > 0 ? tiled_matrix_bytes(m.type, 32, m.ncols) : 0;
    m.w0 = (const uint8_t*)(down ? dn : dual ? gate : up);
    m.w1 = dual ? (const uint8_t*)up : nullptr;
    if (m.type == CHIMERE_TYPE_Q8_0) {   // the copy in operand order
        m.type = kTypeOperand;
        m.w0 = (const uint8_t*)(pw ? (shared ? (down ? pw->sh_down : pw->sh_gu) : (down ? pw->down_exps : pw->gu_exps)) : nullptr);
        m.stride0 = pw && !shared ? (down ? pw->stride_down : pw->stride_gu) : 0;
        m.w1 = nullptr;
        return m;
    }
    if (!shared) { m.stride0 = down ? w->stride_down : dual ? w->stride_gate : w->stride_up; m.stride1 = dual ? w->stride_up : 0; }
    return m;
}

// The expert products of a batch whose routing (ws->offsets, ws->perm) and Q8_1 planes (ws->x_q, ws->x_d, or the packed rows
// of an exchange) are in place: token tiles of every expert with pairs (and of the shared expert; E = 0: of it alone), the
// gate/up GEMM with the activation and the Q8_1 step, the down GEMM; per-pair rows land in ws->pair_out.
static int gemm_experts(const chimere_moe_layer* w, const chimere_moe_prefill_weights* pw, int E, int T, chimere_moe_workspace* ws, cudaStream_t stream,
                        const void* d_packed, int row_bytes, bool mixed, bool mma) {
    if (!ws->prefill_arena) return -1;
    if (w->layout != CHIMERE_LAYOUT_TILED32 || !prefill_dims_ok(w)) return -2;
    const PrefillArena A = prefill_arena(w, ws->max_T);
    if (ws->prefill_bytes < A.total || ((uintptr_t)ws->prefill_arena & 255)) return -4;
    uint8_t* base = (uint8_t*)ws->prefill_arena;
    int32_t* tiles = (int32_t*)(base + A.tiles);
    const Layout L = make_layout(w, ws->max_T);
    const int widest = mixed ? kForwardTileColumns : kTileColumns;
    if (mma) E = 0;   // (the routed experts go elsewhere: tiles of the shared expert alone)
    const int n_tiles_max = E > 0 ? n_tiles_max_for(w, T, widest) : kshared(w) ? (T + 31) / 32 : (T + 127) / 128;
    cudaError_t e = launch_build_tiles(ws->offsets, ws->perm, tiles, mixed ? ws->group_list : nullptr, E, T, w->F_s > 0, mixed ? kForwardGemmPairs : 1, kshared(w), widest, stream);
    if (e != cudaSuccess) return cuda_rc(e);
    // the rows' Q8_1 planes: the workspace's, or (expert-parallel owner) the received packed rows in place
    const int8_t* xq = d_packed ? (const int8_t*)d_packed : ws->x_q;
    const float* xd = d_packed ? (const float*)((const uint8_t*)d_packed + w->H) : ws->x_d;
    const bool sums = kshared(w);   // the shared expert's token tiles carry the blocks' sums
    e = launch_gather_tiles(tiles, ws->perm, xq, d_packed ? row_bytes : w->H, xd, d_packed ? row_bytes / 4 : L.x_d_stride, ws->x_q8, base + A.bx, A.bx_col16,
                            w->H, w->top_k, n_tiles_max, sums, T, stream);
    if (e != cudaSuccess) return cuda_rc(e);
    if (mixed) {   // the small experts: GEMV kernels on the list that the tile builder wrote, per-pair rows only
        const int max_entries = w->E < T * w->top_k ? w->E : T * w->top_k;
        GemvParams gu = gate_up_params(w, T, ws, L);
        gu.nrows_shared = 0; gu.ncols_shared = 0; gu.sh_a = nullptr; gu.sh_b = nullptr; gu.few_tokens = 1;
        e = launch_gate_up_tiled(gu, max_entries, stream);
        if (e != cudaSuccess) return cuda_rc(e);
        GemvParams dn = down_params(w, nullptr, T, ws, L);
        dn.no_combine = 1; dn.few_tokens = 1;
        dn.nrows_shared = 0; dn.ncols_shared = 0; dn.sh_a = nullptr; dn.sh_b = nullptr; dn.split_cols_shared = w->F_s;
        e = launch_down_tiled(dn, max_entries, stream);
        if (e != cudaSuccess) return cuda_rc(e);
    }
    PrefillGemmParams g{};
    g.tiles = tiles; g.perm = ws->perm; g.status = ws->status;
    g.T = T; g.top_k = w->top_k; g.H = w->H;
    for (int down = 0; down < 2 && e == cudaSuccess; ++down) {
        g.shared_sums = sums && !down;
        g.dual = !down && w->act == CHIMERE_ACT_SWIGLU;
        g.m[0] = gemm_mats(w, pw, false, down != 0);
        g.m[1] = gemm_mats(w, pw, true, down != 0);
        if ((E > 0 && !g.m[0].w0) || (w->F_s > 0 && !g.m[1].w0)) return -1;
        g.row_tiles_max = g.m[0].row_tiles > g.m[1].row_tiles ? g.m[0].row_tiles : g.m[1].row_tiles;
        g.b_tiles = base + (down ? A.b2 : A.bx); g.b_col16_bytes = down ? A.b2_col16 : A.bx_col16;
        g.out_tiles = base + A.b2; g.out_col16_bytes = A.b2_col16;
        g.pair_out = ws->pair_out;
        g.shared_out = gemm_shared_rows(w, T, ws);
        if (mixed) {   // sums as the GEMV kernels form them: a token's result does not depend on its batch
            g.inter_q8 = ws->inter_q8; g.inter_stride = (int64_t)L.inter_stride;
            g.inter_q = ws->inter_q; g.inter_q_stride = L.Fmax; g.inter_d = ws->inter_d; g.inter_d_stride = L.inter_d_stride;
            g.as_gemv = 1;
            const int wk = down ? tiled_down_geom(w->type_down, w->F, w->type_sh_down, w->F_s, T).wk
                                : tiled_gate_up_geom(w->type_up, w->type_sh_up, w->H, w->F_s > 0).wk;
            for (PrefillGemmMats& m : g.m) m.slice = m.ncols > 0 ? tiled_slice_units(m.type, m.ncols, wk) / 4 : 1;
        }
        if (mma) {   // the routed experts' products in front; the tiles with minimums alone behind them
            const chimere_moe_layer r = routed_only(w);
            e = down ? launch_mma_down(down_params(&r, nullptr, T, ws, L), ws->offsets, r.E, stream) : launch_mma_gate_up(gate_up_params(&r, T, ws, L), ws->offsets, r.E, stream);
            if (e != cudaSuccess) break;
        }
        e = launch_prefill_gemm(g, down != 0, n_tiles_max, mma, stream);
    }
    return cuda_rc(e);
}

// where the GEMM leaves the shared expert's rows
static float* gemm_shared_rows(const chimere_moe_layer* w, int T, const chimere_moe_workspace* ws) {
    if (kshared(w)) return (float*)((uint8_t*)ws->prefill_arena + prefill_arena(w, ws->max_T).sh_rows);
    return ws->pair_out + (size_t)T * w->top_k * w->H;
}

// routing-weighted sum of every token's pair rows in slot order + the sigmoid-gated shared expert
static cudaError_t finish_tokens(const chimere_moe_layer* w, float* d_y, int T, chimere_moe_workspace* ws, cudaStream_t stream) {
    const float* shared_rows = w->F_s > 0 ? gemm_shared_rows(w, T, ws) : nullptr;
    const float* logit = (w->F_s > 0 && w->shexp_gate_w) ? ws->sh_gate_logit : nullptr;
    return launch_ep_finish(ws->pair_out, nullptr, ws->topk_w, shared_rows, logit, d_y, T, w->H, w->top_k, stream);
}

int chimere_b200_moe_forward_prefill(const chimere_moe_layer* w, const chimere_moe_prefill_weights* pw, const float* d_x, float* d_y,
                                     int T, chimere_moe_workspace* ws, cudaStream_t stream) {
    int rc = check_call(w, d_x, d_y, T, ws, true);
    if (rc) return rc;
    if (!pw || !ws->prefill_arena) return -1;
    // A K-quant shared expert goes through the GEMM with the routed ones where it can (and where the scratch was made for that: its
    // token tiles are larger), else it follows as GEMVs per token.
    const bool ks = kshared(w), gemm = ks && kshared_gemm(w) && pw->sh_gu && pw->sh_down && ws->prefill_bytes >= prefill_arena(w, ws->max_T).total;
    const chimere_moe_layer wr_ = ks && !gemm ? routed_only(w) : *w;
    const chimere_moe_layer* wr = &wr_;
    if (wr->layout != CHIMERE_LAYOUT_TILED32 || !prefill_dims_ok(wr)) return -2;
    const chimere_moe_layer route_ = ks ? routed_only(w) : *w;
    if (ws->prefill_bytes < prefill_arena(wr, ws->max_T).total || ((uintptr_t)ws->prefill_arena & 255)) return -4;
    if (prefill_as_decode(&route_, T)) return chimere_b200_moe_forward(w, d_x, d_y, T, ws, stream);
    RouteParams rp = route_params(&route_, d_x, T, ws, ks);
    rp.list_mode = 2;   // no work entries: the kernels make their own tiles
    cudaError_t e = launch_route(rp, stream);
    if (e != cudaSuccess) return cuda_rc(e);
    const bool mma = prefill_mma(&route_, T) && mma_runs(&route_, T, ws);
    rc = mma && !gemm ? run_mma(&route_, T, ws, stream) : gemm_experts(wr, pw, wr->E, T, ws, stream, nullptr, 0, false, mma);
    if (rc) return rc;
    e = finish_tokens(wr, d_y, T, ws, stream);
    if (e != cudaSuccess || !ks || gemm) return cuda_rc(e);
    return kshared_chain(w, T, d_y, ws, stream);
}

// Expert-parallel owner rank, prefill-size: as chimere_b200_moe_experts, with the local experts on the grouped GEMM.
int chimere_b200_moe_experts_prefill(const chimere_moe_layer* w_local, const chimere_moe_prefill_weights* pw_local, int n_rows,
                                     chimere_moe_workspace* ws, cudaStream_t stream) {
    if (n_rows == 0) return 0;
    int rc = check_call(w_local, ws, ws, n_rows, ws);
    if (rc) return rc;
    if (w_local->layout != CHIMERE_LAYOUT_TILED32 || w_local->top_k != 1 || w_local->F_s != 0) return -2;
    RouteParams p = route_params(w_local, nullptr, n_rows, ws);
    p.has_shared = 0;
    p.list_mode = 2;
    cudaError_t e = launch_permute(p, stream);
    if (e != cudaSuccess) return cuda_rc(e);
    if (!pw_local) return -1;
    return gemm_experts(w_local, pw_local, w_local->E, n_rows, ws, stream);
}

// Expert-parallel home rank, prefill-size: the shared expert of this rank's T tokens on the grouped GEMM (token tiles of
// the shared expert only), per-token rows into ws->pair_out[T * top_k + t] as chimere_b200_moe_shared_expert leaves them.
int chimere_b200_moe_shared_expert_prefill(const chimere_moe_layer* w, const chimere_moe_prefill_weights* pw, int T, chimere_moe_workspace* ws,
                                           cudaStream_t stream) {
    int rc = check_call(w, ws, ws, T, ws);
    if (rc) return rc;
    if (w->F_s <= 0) return 0;
    if (!pw || !ws->prefill_arena) return -1;
    return gemm_experts(w, pw, 0, T, ws, stream);   // (no routed expert gets a tile)
}

// ... with the rows where an exchange left them: packed rows [H int8][d_stride f32][int32 local expert id] (see ep_pack).
int chimere_b200_moe_experts_packed_prefill(const chimere_moe_layer* w_local, const chimere_moe_prefill_weights* pw_local, int n_rows,
                                            const void* d_rows, int row_bytes, chimere_moe_workspace* ws, cudaStream_t stream) {
    if (n_rows == 0) return 0;
    if (!d_rows) return -1;
    int rc = check_call(w_local, ws, ws, n_rows, ws);
    if (rc) return rc;
    if (w_local->layout != CHIMERE_LAYOUT_TILED32 || w_local->top_k != 1 || w_local->F_s != 0) return -2;
    const int ds = (w_local->H / 32 + 3) & ~3;
    if (row_bytes % 16 || row_bytes < w_local->H + 4 * ds + 4) return -2;
    RouteParams p = route_params(w_local, nullptr, n_rows, ws);
    p.has_shared = 0;
    p.list_mode = 2;
    p.topk_idx = (int32_t*)((uint8_t*)d_rows + w_local->H + 4 * ds);
    p.idx_stride = row_bytes / 4;
    cudaError_t e = launch_permute(p, stream);
    if (e != cudaSuccess) return cuda_rc(e);
    if (!pw_local) return -1;
    return gemm_experts(w_local, pw_local, w_local->E, n_rows, ws, stream, d_rows, row_bytes);
}

int chimere_b200_moe_ep_pack_sorted(const chimere_moe_layer* w, int T, chimere_moe_workspace* ws, void* d_send, int32_t* d_slot,
                                    int experts_per_rank, int row_bytes, cudaStream_t stream) {
    int rc = check_call(w, d_send, d_slot, T, ws);
    if (rc) return rc;
    const int ds = (w->H / 32 + 3) & ~3;
    if (experts_per_rank <= 0 || row_bytes % 16 || row_bytes < w->H + 4 * ds + 4) return -2;
    return cuda_rc(launch_ep_pack_sorted(ws->perm, ws->topk_idx, ws->x_q, ws->x_d, ds, (uint8_t*)d_send, d_slot, T, w->top_k, w->H,
                                         experts_per_rank, row_bytes, stream));
}

int chimere_b200_moe_forward_residual_norm(const chimere_moe_layer* w, const chimere_moe_prefill_weights* pw, const float* d_hidden,
                                           float* d_residual, const float* d_norm_weight, float eps, float* d_y, int T,
                                           chimere_moe_workspace* ws, cudaStream_t stream) {
    int rc = check_call(w, d_hidden, d_y, T, ws, true);
    if (rc) return rc;
    if (!d_residual || !d_norm_weight || !ws->pair_out) return -1;
    if (!pw && pairs_forward(w, T, ws)) {
        const chimere_moe_layer wr = kshared(w) ? routed_only(w) : *w;
        if (route_norm_runs(route_params(&wr, nullptr, T, ws))) return run_pairs(w, nullptr, d_hidden, d_residual, d_norm_weight, eps, d_y, T, ws, stream);
    }
    // the normalised rows live in the first T rows of the per-pair output area until the router and the Q8_1 step have
    // read them; the down stage writes that area only afterwards
    float* normed = ws->pair_out;
    cudaError_t e = launch_add_residual_rmsnorm(d_hidden, d_residual, d_norm_weight, normed, T, w->H, eps, stream);
    if (e != cudaSuccess) return cuda_rc(e);
    return pw ? chimere_b200_moe_forward_prefill(w, pw, normed, d_y, T, ws, stream) : chimere_b200_moe_forward(w, normed, d_y, T, ws, stream);
}

int chimere_b200_moe_routing_trace(const chimere_moe_layer* w, int T, const chimere_moe_workspace* ws, uint8_t* d_trace,
                                   int32_t* d_expert_load, cudaStream_t stream) {
    if (!w || !ws || !ws->topk_idx || !d_trace) return -1;
    if (T <= 0 || T > ws->max_T || w->top_k <= 0 || w->top_k > kMaxTopK || w->E <= 0 || w->E > kMaxExperts) return -2;
    return cuda_rc(launch_routing_trace(ws->topk_idx, d_trace, d_expert_load, T, w->top_k, w->E, stream));
}

int chimere_b200_rmsnorm(const float* d_x, float* d_y, int T, int H, float eps, cudaStream_t stream) {
    if (!d_x || !d_y) return -1;
    if (T < 0 || H <= 0) return -2;
    return cuda_rc(launch_rmsnorm(d_x, d_y, T, H, eps, stream));
}

// ---------------------------------------------------------------- legacy operator entries --
void chimere_quantize_q8_1(const float* input, void* output, int64_t ncols, int64_t ncols_padded, cudaStream_t stream) {
    launch_quantize_q8_1(input, output, ncols, ncols_padded, 1, stream);
}
void chimere_quantize_q8_1_batched(const float* input, void* output, int64_t ncols, int64_t ncols_padded, int batch,
                                   cudaStream_t stream) {
    launch_quantize_q8_1(input, output, ncols, ncols_padded, batch, stream);
}
void chimere_mmvq_iq3s(const void* weights, const void* input_q8, float* output, int ncols, int nrows, int, cudaStream_t stream) {
    launch_mmvq(CHIMERE_TYPE_IQ3_S, weights, input_q8, output, nullptr, ncols, nrows, 0, 0, 1, stream);
}
void chimere_mmvq_q8_0(const void* weights, const void* input_q8, float* output, int ncols, int nrows, int, cudaStream_t stream) {
    launch_mmvq(CHIMERE_TYPE_Q8_0, weights, input_q8, output, nullptr, ncols, nrows, 0, 0, 1, stream);
}
void chimere_mmvq_q4_0(const void* weights, const void* input_q8, float* output, int ncols, int nrows, int, cudaStream_t stream) {
    launch_mmvq(CHIMERE_TYPE_Q4_0, weights, input_q8, output, nullptr, ncols, nrows, 0, 0, 1, stream);
}
// Fused quantize + GEMV from an f32 input row (ffi/ggml_cuda_gemv.cu:322-352): Q8_1 of the input into the caller's
// scratch (pad(ncols, 512) / 32 * 36 bytes, blocks past ncols zero), then the GEMV above on that scratch.
static void mmvq_f32(int wtype, const void* weights, const float* input_f32, float* output, int ncols, int nrows, int ncols_padded,
                     void* q8_scratch, cudaStream_t stream) {
    launch_quantize_q8_1(input_f32, q8_scratch, ncols, ncols_padded, 1, stream);
    launch_mmvq(wtype, weights, q8_scratch, output, nullptr, ncols, nrows, 0, 0, 1, stream);
}
void chimere_mmvq_iq3s_f32(const void* weights, const float* input_f32, float* output, int ncols, int nrows, int ncols_padded,
                           void* q8_scratch, cudaStream_t stream) {
    mmvq_f32(CHIMERE_TYPE_IQ3_S, weights, input_f32, output, ncols, nrows, ncols_padded, q8_scratch, stream);
}
void chimere_mmvq_q8_0_f32(const void* weights, const float* input_f32, float* output, int ncols, int nrows, int ncols_padded,
                           void* q8_scratch, cudaStream_t stream) {
    mmvq_f32(CHIMERE_TYPE_Q8_0, weights, input_f32, output, ncols, nrows, ncols_padded, q8_scratch, stream);
}
void chimere_mmvq_q4_0_f32(const void* weights, const float* input_f32, float* output, int ncols, int nrows, int ncols_padded,
                           void* q8_scratch, cudaStream_t stream) {
    mmvq_f32(CHIMERE_TYPE_Q4_0, weights, input_f32, output, ncols, nrows, ncols_padded, q8_scratch, stream);
}
void chimere_mmvq_q5k(const void* weights, const void* input_q8, float* output, int ncols, int nrows, int, cudaStream_t stream) {
    launch_mmvq_kquant(CHIMERE_TYPE_Q5_K, weights, input_q8, output, ncols, nrows, stream);
}
void chimere_mmvq_q4k(const void* weights, const void* input_q8, float* output, int ncols, int nrows, int, cudaStream_t stream) {
    launch_mmvq_kquant(CHIMERE_TYPE_Q4_K, weights, input_q8, output, ncols, nrows, stream);
}
void chimere_mmvq_q6k(const void* weights, const void* input_q8, float* output, int ncols, int nrows, int, cudaStream_t stream) {
    launch_mmvq_kquant(CHIMERE_TYPE_Q6_K, weights, input_q8, output, ncols, nrows, stream);
}
static void mmvq_kquant_f32(int wtype, const void* weights, const float* input_f32, float* output, int ncols, int nrows, int ncols_padded,
                            void* q8_scratch, cudaStream_t stream) {
    launch_quantize_q8_1(input_f32, q8_scratch, ncols, ncols_padded, 1, stream);
    launch_mmvq_kquant(wtype, weights, q8_scratch, output, ncols, nrows, stream);
}
void chimere_mmvq_q5k_f32(const void* weights, const float* input_f32, float* output, int ncols, int nrows, int ncols_padded,
                          void* q8_scratch, cudaStream_t stream) {
    mmvq_kquant_f32(CHIMERE_TYPE_Q5_K, weights, input_f32, output, ncols, nrows, ncols_padded, q8_scratch, stream);
}
void chimere_mmvq_q4k_f32(const void* weights, const float* input_f32, float* output, int ncols, int nrows, int ncols_padded,
                          void* q8_scratch, cudaStream_t stream) {
    mmvq_kquant_f32(CHIMERE_TYPE_Q4_K, weights, input_f32, output, ncols, nrows, ncols_padded, q8_scratch, stream);
}
void chimere_mmvq_q6k_f32(const void* weights, const float* input_f32, float* output, int ncols, int nrows, int ncols_padded,
                          void* q8_scratch, cudaStream_t stream) {
    mmvq_kquant_f32(CHIMERE_TYPE_Q6_K, weights, input_f32, output, ncols, nrows, ncols_padded, q8_scratch, stream);
}
void chimere_mmvq_iq3s_batched(const void* all_weights, const void* input_q8, float* output, const int* expert_ids, int ncols,
                               int nrows, int, int64_t expert_stride, int64_t input_stride, int top_k, cudaStream_t stream) {
    launch_mmvq(CHIMERE_TYPE_IQ3_S, all_weights, input_q8, output, expert_ids, ncols, nrows, expert_stride, input_stride, top_k, stream);
}
void chimere_mmvq_q4_0_batched(const void* all_weights, const void* input_q8, float* output, const int* expert_ids, int ncols,
                               int nrows, int, int64_t expert_stride, int64_t input_stride, int top_k, cudaStream_t stream) {
    launch_mmvq(CHIMERE_TYPE_Q4_0, all_weights, input_q8, output, expert_ids, ncols, nrows, expert_stride, input_stride, top_k, stream);
}
void chimere_mmvq_q8_0_batched(const void* all_weights, const void* input_q8, float* output, const int* expert_ids, int ncols,
                               int nrows, int, int64_t expert_stride, int64_t input_stride, int top_k, cudaStream_t stream) {
    launch_mmvq(CHIMERE_TYPE_Q8_0, all_weights, input_q8, output, expert_ids, ncols, nrows, expert_stride, input_stride, top_k, stream);
}
int chimere_q8_1_block_bytes(void) { return kQ81Bytes; }
int chimere_q8_1_block_elems(void) { return 32; }
int chimere_matrix_row_padding(void) { return 512; }

}  // extern "C"
