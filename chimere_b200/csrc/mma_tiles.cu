// mma_tiles.cu -- expert products of batches whose experts hold a few tokens to a few dozen: 16 pairs of one expert at a time on the
// warp-level int8 MMA (m16n8k32), weights from the tiled32 form straight into its fragments.
//
// A tile of 16 columns asks little of a tensor pipe, and much of what stands around it: on the tcgen05 kernel (gemm_i8.cu) every packed
// byte is expanded to shared memory, every accumulator comes back from TMEM, and each of 24 warps keeps step with rings and barriers
// (2 800 warp instructions per 128 rows x 128 columns of weights and 16 tokens).  Here a warp owns 32 rows of one matrix and a slice of K: the
// row's nibbles become the A operand in the registers that the load wrote, the accumulators appear in registers, and nothing is
// exchanged until a slice is done (1 500 with up to eight columns, half of it outside the products).  The MMA starts from 2^19 so that an accumulator's bits are a positive denormal float:
// no integer-to-float step (see readback_tile in gemm_i8.cu).
//
//   work   : token tile = up to 16 pairs of one expert (or tokens of the shared one), from the dispatch step's offsets, no list;
//            item = token tile x as many 32-row tiles as 16 warps hold (matrices x row tiles x K slices); a CTA takes a run
//            of consecutive items, so that it stays on a token tile for most of its rows
//   tokens : Q8_1 planes of a tile's columns in shared memory, two buffers: the next tile's come in (cp.async) during this tile's last item
//   weights: a group of four units in registers, every unit asked for again as soon as it is decoded, for the next group or the next item
//   sums   : the K slices of an item meet in shared memory; a column of it is added up, activated and stored by one warp, another one
//            for every item, and nobody waits for that but for the buffer, two items later
//
// Sums are bit for bit those of bulk_kernel (gemv_tiled.cu): exact block dots, the same products in the same order, K slices added in order.
//
// What bounds it: the latency of the weights (37 KB in flight per SM) and the instructions around the products, half and half (52 % of
// the issue slots busy, DRAM at 2.9 TB/s in the gate/up launch of 64 uniform tokens, 256 experts; 85 us, the expert GEMVs and the GEMM
// before 130).  Layer, us: 64 tokens 191 -> 145 (61 of skewed routing 115 -> 71), 128 in the prefill entry 254 -> 175; 128 wide experts, 48 tokens
// 291 -> 236.  Tried: two groups in flight (registers spill: 154 instead of 145), weights through a ring of bulk copies in shared memory (182: a
// copy and a wait per group cost more than they save), a CTA barrier per item instead of the column's one warp (162), equal numbers of items
// per CTA (176).
#include "common.cuh"
#include "kernels.h"
#include "tiled.cuh"

namespace chimere {

constexpr int kMmaCols = 16, kMmaWarps = 16, kMmaThreads = 32 * kMmaWarps;
constexpr int kMmaRedPitch = 36;                        // floats per column of a 32-row block of sums: the lanes of a store on different banks
constexpr int kMmaRedWarp = kMmaCols * kMmaRedPitch;
constexpr uint32_t kMmaRowBits = 0x71800000u;           // 2^100 (as in gemm_i8.cu: the dot comes out times 2^-49)
constexpr uint32_t kMmaOffsetBits = 0xB0800000u;        // -2^19 * 2^-149 * 2^100

__device__ __forceinline__ void mma_s8(uint32_t (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(1u << 19));
}
__device__ __forceinline__ void ldsm_x4(uint32_t a, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(a));
}
__device__ __forceinline__ void ldsm_x2(uint32_t a, uint32_t& r0, uint32_t& r1) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(a));
}
__device__ __forceinline__ void lds_2x64(uint32_t a, uint64_t& x, uint64_t& y) { asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"(a)); }
__device__ __forceinline__ uint64_t lds_1x64(uint32_t a) { uint64_t x; asm volatile("ld.shared.b64 %0, [%1];" : "=l"(x) : "r"(a)); return x; }
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void ldg32(uint32_t& v, const uint8_t* a) { asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(a)); }
__device__ __forceinline__ void ldg16(uint16_t& v, const uint8_t* a) { asm volatile("ld.global.nc.L1::no_allocate.u16 %0, [%1];" : "=h"(v) : "l"(a)); }

// Four units of a 32-row tile: word [u][i] = bytes 4 * (lane & 3) .. of row (lane >> 2) + 8 i, i.e. what the MMA's A fragments hold
// of the low and of the high nibbles; scales of row `lane`.
template <int TYPE> struct MmaGroup;
template <> struct MmaGroup<CHIMERE_TYPE_Q4_0> {
    uint32_t w[4][4];
    uint16_t d[4];
    __device__ static __forceinline__ uint32_t offset(int g, int lane) { return (uint32_t)(g * 2304 + lane * 4); }
    template <bool ALL>
    __device__ __forceinline__ void load_unit(int u, const uint8_t* gp, const uint8_t* sp, int on) {
#pragma unroll
        for (int i = 0; i < 4; ++i) { if (ALL) ldg32(w[u][i], gp + u * 576 + i * 128); else ldg32_if(w[u][i], gp + u * 576 + i * 128, on); }
        if (ALL) ldg16(d[u], sp + u * 576); else ldg16_if(d[u], sp + u * 576, on);
    }
    __device__ static __forceinline__ const uint8_t* scales(const uint8_t* gp, int, int lane) { return gp - lane * 2 + 512; }
    __device__ __forceinline__ void load_scales(const uint8_t*, int) {}
};
template <> struct MmaGroup<CHIMERE_TYPE_IQ3_S> {
    uint32_t w[4][4];
    uint16_t d;
    uint32_t sc;
    __device__ static __forceinline__ uint32_t offset(int g, int lane) { return (uint32_t)((g >> 1) * 4288 + (g & 1) * 2048 + lane * 4); }
    template <bool ALL>
    __device__ __forceinline__ void load_unit(int u, const uint8_t* gp, const uint8_t*, int on) {
#pragma unroll
        for (int i = 0; i < 4; ++i) { if (ALL) ldg32(w[u][i], gp + u * 512 + i * 128); else ldg32_if(w[u][i], gp + u * 512 + i * 128, on); }
    }
    __device__ static __forceinline__ const uint8_t* scales(const uint8_t* gp, int g, int) { return gp + (4096 - (g & 1) * 2048); }
    __device__ __forceinline__ void load_scales(const uint8_t* sp, int on) {
        ldg16_if(d, sp - (threadIdx.x & 31) * 2, on);
        ldg32_if(sc, sp + 64, on);
    }
};

template <int TYPE>
__device__ __forceinline__ void fill_group(MmaGroup<TYPE>& r, const uint8_t* tile, int g, int nu, int lane) {
    const uint8_t* gp = tile + MmaGroup<TYPE>::offset(g, lane);
    const uint8_t* sp = MmaGroup<TYPE>::scales(gp, g, lane);
#pragma unroll
    for (int u = 0; u < kGroupUnits; ++u) r.template load_unit<false>(u, gp, sp, u < nu);
    r.load_scales(sp, nu > 0);
}

// One group (units u < nu) against the tile's columns (8 or, TWO, 16 of them); b: shared address of the warp's ldmatrix rows at the
// group's first unit, s: of the lane's four column scales there.  acc carries 2^-49 (Q4_0: 2^-45).  The registers are asked for again at
// group gn of tile np: ALL four units there (and here), else nn of them.
template <int TYPE, bool TWO, bool ALL>
__device__ __forceinline__ void mma_group(MmaGroup<TYPE>& r, int g, int nu, uint32_t b, uint32_t s, uint64_t (&acc)[4][2], const uint8_t* np, int gn, int nn, int lane) {
    constexpr bool kGroup = TYPE == CHIMERE_TYPE_IQ3_S;
    constexpr uint32_t kOdd = kGroup ? 0x08080808u : 0u;   // 8 * (2c + 1) = 16c + 8
    constexpr int kT = TWO ? 2 : 1;
    const int quad = lane >> 2;
    uint32_t sd[4][2], ss[4];
    if constexpr (kGroup) {
        const uint32_t sc = r.sc >> (16 * (g & 1));
#pragma unroll
        for (int i = 0; i < 4; ++i) { ss[i] = __shfl_sync(0xffffffffu, sc, quad + 8 * i); sd[i][0] = __shfl_sync(0xffffffffu, (uint32_t)r.d, quad + 8 * i); }
    } else {
        const uint32_t p0 = (uint32_t)r.d[0] | ((uint32_t)r.d[1] << 16), p1 = (uint32_t)r.d[2] | ((uint32_t)r.d[3] << 16);
#pragma unroll
        for (int i = 0; i < 4; ++i) { sd[i][0] = __shfl_sync(0xffffffffu, p0, quad + 8 * i); sd[i][1] = __shfl_sync(0xffffffffu, p1, quad + 8 * i); }
    }
    const uint8_t* gp = np + MmaGroup<TYPE>::offset(gn, lane);
    const uint8_t* sp = MmaGroup<TYPE>::scales(gp, gn, lane);
    uint64_t part[4][kT];
    if constexpr (kGroup) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int t = 0; t < kT; ++t) part[i][t] = 0ull;
    }
#pragma unroll
    for (int u = 0; u < kGroupUnits; ++u) {
        if (ALL || u < nu) {
            uint32_t bq[4];
            if (TWO) ldsm_x4(b + u * 32, bq[0], bq[1], bq[2], bq[3]);
            else ldsm_x2(b + u * 32, bq[0], bq[1]);
            uint64_t x[kT];
            if constexpr (TWO) lds_2x64(s + u * 64, x[0], x[1]);
            else x[0] = lds_1x64(s + u * 64);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t d[kT][4];
                const uint32_t w0 = r.w[u][2 * h], w1 = r.w[u][2 * h + 1];
                const uint32_t a0 = ((w0 << 4) & 0xF0F0F0F0u) ^ (0x80808080u | kOdd), a1 = ((w1 << 4) & 0xF0F0F0F0u) ^ (0x80808080u | kOdd);
                const uint32_t a2 = (w0 & 0xF0F0F0F0u) | kOdd, a3 = (w1 & 0xF0F0F0F0u) | kOdd;
#pragma unroll
                for (int t = 0; t < kT; ++t) mma_s8(d[t], a0, a1, a2, a3, bq[2 * t], bq[2 * t + 1]);
                if (h == 1) r.template load_unit<ALL>(u, gp, sp, u < nn);
#pragma unroll
              for (int q = 0; q < 2; ++q) {
                const int i = 2 * h + q;   // row quad + 8 i
                uint64_t r2, o2, f2;
                if constexpr (kGroup) {
                    // 1 + 2 * sub-scale, times 2^97 and times what takes the offset out again, from the bits of 2^23 + sub-scale
                    const float f = __uint_as_float(((ss[i] >> (4 * u)) & 15u) | 0x4B000000u);
                    const float kr = fmaf(f, 0x1p98f, 0x1p97f - 0x1p121f), ko = fmaf(f, -0x1p-32f, 0x1p-9f - 0x1p-33f);
                    r2 = pack2f(kr, kr); o2 = pack2f(ko, ko);
                } else {
                    const float dw = h2f(sd[i][u >> 1] >> (16 * (u & 1)));
                    f2 = pack2f(dw, dw);
                    r2 = pack2(kMmaRowBits, kMmaRowBits); o2 = pack2(kMmaOffsetBits, kMmaOffsetBits);
                }
#pragma unroll
                for (int t = 0; t < kT; ++t) {
                    const uint64_t v = fma2(pack2(d[t][2 * q], d[t][2 * q + 1]), r2, o2);   // exact
                    if constexpr (kGroup) part[i][t] = fma2(v, x[t], part[i][t]);
                    else acc[i][t] = fma2(mul2(f2, x[t]), v, acc[i][t]);
                }
              }
            }
        } else r.template load_unit<ALL>(u, gp, sp, u < nn);
    }
    r.load_scales(sp, ALL || nn > 0);
    if constexpr (kGroup) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float dw = h2f(sd[i][0]);
            const uint64_t f2 = pack2f(dw, dw);
#pragma unroll
            for (int t = 0; t < kT; ++t) acc[i][t] = fma2(f2, part[i][t], acc[i][t]);
        }
    }
}

// An item's groups by one warp: w this item's tile (nu units from group g0), nw the next one's (xnu units from unit xu0).
template <int TYPE, bool TWO, int D>
__device__ __forceinline__ void mma_item(MmaGroup<TYPE> (&ring)[D], const uint8_t* w, const uint8_t* nw, int g0, int nu, int xu0, int xnu, uint32_t b0, uint32_t s0,
                                         uint64_t (&acc)[4][2], int lane) {
    const int ng = (nu + 3) >> 2;
    for (int gg = 0; gg < ng; gg += D) {
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const int g = gg + d;
            if (g < ng) {
                const bool same = g + D < ng;
                const int n = min(4, nu - 4 * g), nn = same ? min(4, nu - 4 * (g + D)) : max(0, min(4, xnu - 4 * d));
                const uint8_t* np = same ? w : nw;
                const int gn = same ? g0 + g + D : (xu0 >> 2) + d;
                if (n == 4 && nn == 4) mma_group<TYPE, TWO, true>(ring[d], g0 + g, n, b0 + g * 128, s0 + g * 256, acc, np, gn, nn, lane);
                else mma_group<TYPE, TWO, false>(ring[d], g0 + g, n, b0 + g * 128, s0 + g * 256, acc, np, gn, nn, lane);
            }
        }
    }
}

struct MmaGeom { int wk, wr, slice_r, slice_s, pitch, nb_max; };   // K slices, row tiles per item, units per slice, bytes of a column's row in shared memory

__host__ __device__ inline size_t mma_tile_bytes(int pitch, int nb_max) { return (size_t)kMmaCols * pitch + (size_t)nb_max * 64; }

// Stage 0: act(gate . x, up . x) -> Q8_1 of the intermediates; stage 1: down . intermediates -> per-pair rows.
template <int TYPE, int STAGE, bool DUAL, int D>
__global__ void __launch_bounds__(kMmaThreads, 1) mma_tile_kernel(const __grid_constant__ GemvParams p, const int32_t* offsets, int E, const __grid_constant__ MmaGeom geo) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ int s_first[257], s_load[257], s_off[257], s_scan[16];
    __shared__ int s_prow[2][kMmaCols];
    __shared__ int4 s_tile[2];
    __shared__ __align__(8) uint64_t s_full[2], s_empty[2];   // an item's sums are there / have been read
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int T = p.T, k = p.top_k, P = T * k;
    const uint32_t tile_bytes_s = (uint32_t)mma_tile_bytes(geo.pitch, geo.nb_max);
    float* red = reinterpret_cast<float*>(smem + 2 * tile_bytes_s);   // [2][warp][16 columns][36]
    // this warp: matrix, row tile within the item, K slice
    const int wk = geo.wk, wr = geo.wr, s_id = warp % wk, rt_id = warp / wk % wr, mat = warp / (wk * wr);

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], kMmaWarps); mbar_init(&s_empty[i], kMmaWarps); }
        mbar_fence_init();
    }
    griddep_wait();
    if (tid == 0) griddep_launch();
    // first token tile of every expert
    if (tid < 256) {
        const int o = tid < E ? __ldcg(offsets + tid) : 0, cnt = tid < E ? __ldcg(offsets + tid + 1) - o : 0, n = (cnt + kMmaCols - 1) / kMmaCols;
        const int own = n > 0 ? 3 * (n - 1) + (cnt - (n - 1) * kMmaCols > 8 ? 3 : 2) : 0;
        int incl = n, incl_l = own;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, incl, s), b = __shfl_up_sync(0xffffffffu, incl_l, s);
            if (lane >= s) { incl += a; incl_l += b; }
        }
        if (lane == 31) { s_scan[warp] = incl; s_scan[8 + warp] = incl_l; }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        int base = 0, base_l = 0, total = 0, total_l = 0;
        for (int w = 0; w < 8; ++w) {
            if (w < warp) { base += s_scan[w]; base_l += s_scan[8 + w]; }
            total += s_scan[w]; total_l += s_scan[8 + w];
        }
        s_first[tid] = base + incl - n;
        s_load[tid] = base_l + incl_l - own;
        if (tid < E) s_off[tid] = o;
        if (tid == 0) { s_first[256] = total; s_load[256] = total_l; s_off[E] = __ldcg(offsets + E); }
    }
    __syncthreads();
    const int rows32_r = p.nrows_routed >> 5, rows32_s = p.nrows_shared >> 5;
    const int rg_r = (rows32_r + wr - 1) / wr, rg_s = (rows32_s + wr - 1) / wr;
    const int n_sh = p.nrows_shared > 0 ? (T + kMmaCols - 1) / kMmaCols : 0, items_s = n_sh * rg_s;
    // This CTA's run of items, the shared expert's first.  An item of more than eight columns counts for three, the others for two (about
    // what they take; the shared expert's by the length of its rows): with equal numbers of items the CTAs that have the shared expert's
    // were a third behind at 64 tokens of uniform routing.
    const int each_s = n_sh > 0 ? max(1, 3 * p.ncols_shared / p.ncols_routed) : 1;
    const int64_t load_s = each_s * (int64_t)items_s, load = load_s + (int64_t)s_load[256] * rg_r;
    auto item_at = [&](int64_t x) {
        if (x < load_s) return (int)(x / each_s);
        x -= load_s;
        int lo = 0, hi = 256;   // the expert that x falls into
        while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if ((int64_t)s_load[mid] * rg_r <= x) lo = mid; else hi = mid; }
        const int tiles = s_first[lo + 1] - s_first[lo];
        const int64_t in = x - (int64_t)s_load[lo] * rg_r, full = 3 * (int64_t)max(tiles - 1, 0) * rg_r;
        const int each = s_load[lo + 1] - s_load[lo] - 3 * (tiles - 1);   // the last tile's
        return items_s + s_first[lo] * rg_r + (int)min(in < full ? in / 3 : full / 3 + (in - full) / max(each, 1), (int64_t)tiles * rg_r);
    };
    int item = item_at(load * blockIdx.x / gridDim.x);
    const int item_end = blockIdx.x + 1 == gridDim.x ? items_s + s_first[256] * rg_r : item_at(load * (blockIdx.x + 1) / gridDim.x);
    if (item >= item_end) return;

    // A token tile: { expert or -1 = shared, first pair (or token), columns, row groups }, kept in shared memory (registers are what these
    // kernels are short of); every warp writes the same words before it reads them.
    auto find_tile = [&](int it, int b) {   // -> row group of item `it` in its tile
        int4 t;
        int rg;
        if (it < items_s) {
            const int j = it / rg_s;
            rg = it - j * rg_s;
            t = make_int4(-1, j * kMmaCols, min(kMmaCols, T - j * kMmaCols), rg_s);
        } else {
            const int j = (it - items_s) / rg_r;
            rg = it - items_s - j * rg_r;
            int lo = 0, hi = E;   // s_first[lo] <= j < s_first[hi]
            while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (s_first[mid] <= j) lo = mid; else hi = mid; }
            const int start = s_off[lo] + (j - s_first[lo]) * kMmaCols;
            t = make_int4(lo, start, min(kMmaCols, s_off[lo + 1] - start), rg_r);
        }
        if (lane == 0) s_tile[b] = t;
        __syncwarp();
        return rg;
    };
    // the output row of column `warp` of a tile (its pair, or the shared expert's row of a token)
    auto row_of = [&](int b) { const int4 t = s_tile[b]; return warp < t.z ? (t.x < 0 ? P + t.y + warp : __ldcg(p.perm + t.y + warp)) : 0; };
    // columns of a tile on their way to their buffer: warp = column
    auto fetch = [&](int b, int prow) {
        const int4 t = s_tile[b];
        if (warp < t.z) {
            const int ncols = t.x < 0 ? p.ncols_shared : p.ncols_routed;
            const int row = STAGE == 0 ? (t.x < 0 ? t.y + warp : prow / k) : prow;
            const uint32_t dst = smem_u32(smem) + b * tile_bytes_s + (uint32_t)warp * geo.pitch;
            const int8_t* q = p.in_soa_q + (size_t)row * p.in_soa_q_stride;
            for (int c = lane; c < ncols >> 4; c += 32) cp_async16(dst + c * 16, q + c * 16);
            const float* d = p.in_soa_d + (size_t)row * p.in_soa_d_stride;
            // scales: [unit][lane of a quad][two column pairs]
            const uint32_t sdst = smem_u32(smem) + b * tile_bytes_s + (uint32_t)(kMmaCols * geo.pitch) + ((warp & 7) >> 1) * 16 + (warp >> 3) * 8 + (warp & 1) * 4;
            for (int c = lane; c < ncols >> 5; c += 32) cp_async4(sdst + c * 64, d + c);
            if (lane == 0) s_prow[b][warp] = prow;
        }
    };
    // weights of row group rg of a tile: this warp's row tile of its matrix (null: behind the last row), and its slice of K
    auto weights = [&](int b, int rg) -> const uint8_t* {
        const int expert = s_tile[b].x, tile = rg * wr + rt_id;
        const bool sh = expert < 0;
        if (tile >= (sh ? rows32_s : rows32_r)) return nullptr;
        const int64_t tb = Tiled<TYPE>::tile_bytes(sh ? p.ncols_shared : p.ncols_routed);
        const uint8_t* m;
        if (STAGE == 0 && !(DUAL && mat == 1)) m = sh ? p.sh_b : p.w_b + (size_t)expert * p.stride_b;   // up
        else m = sh ? p.sh_a : p.w_a + (size_t)expert * p.stride_a;                                      // gate, down
        return m + (size_t)tile * tb;
    };
    auto slice = [&](int b, int& u0, int& nu) {
        const bool sh = s_tile[b].x < 0;
        const int nb = (sh ? p.ncols_shared : p.ncols_routed) >> 5, per = sh ? geo.slice_s : geo.slice_r;
        u0 = min(nb, s_id * per); nu = min(nb, u0 + per) - u0;
    };

    int buf = 0, rg = find_tile(item, 0);
    fetch(0, row_of(0));
    int u0, nu;
    slice(0, u0, nu);
    const uint8_t* w = weights(0, rg);
    MmaGroup<TYPE> ring[D];
#pragma unroll
    for (int d = 0; d < D; ++d) fill_group<TYPE>(ring[d], w, (u0 >> 2) + d, w ? max(0, min(4, nu - 4 * d)) : 0, lane);
    int step = 0;
    while (true) {
        // ---- a token tile: its rows are on their way to `buf` ----
        const int tile_end = min(item_end, item + s_tile[buf].w - rg);
        const bool next_tile = tile_end < item_end;
        int nprow = 0;
        cp_async_wait();
        __syncthreads();   // (everybody is done with the other buffer, too)
        if (next_tile) { find_tile(tile_end, buf ^ 1); nprow = row_of(buf ^ 1); }
        const uint32_t b_tile = smem_u32(smem) + buf * tile_bytes_s;
        const int cols = s_tile[buf].z;
        const bool two = cols > 8;
        // ldmatrix rows: lane l names 16 bytes of column (l >> 4) * 8 + (l & 7), K half (l >> 3) & 1
        const uint32_t b0 = b_tile + (uint32_t)(((two ? lane >> 4 : 0) * 8 + (lane & 7)) * geo.pitch + ((lane >> 3) & 1) * 16) + (uint32_t)u0 * 32;
        const uint32_t s0 = b_tile + (uint32_t)(kMmaCols * geo.pitch) + (lane & 3) * 16 + (uint32_t)u0 * 64;
        for (; item < tile_end; ++item, ++step) {
            const bool last = item + 1 == tile_end, more = !last || next_tile;
            if (last && more) fetch(buf ^ 1, nprow);
            // the item behind: its weights, its slice
            const uint8_t* nw = !more ? nullptr : last ? weights(buf ^ 1, 0) : weights(buf, rg + 1);
            int xu0 = u0, xnu = nu;
            if (last && more) slice(buf ^ 1, xu0, xnu);
            if (!nw) xnu = 0;
            uint64_t acc[4][2];
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0ull;
            if (w) {
                if (two) mma_item<TYPE, true>(ring, w, nw, u0 >> 2, nu, xu0, xnu, b0, s0, acc, lane);
                else mma_item<TYPE, false>(ring, w, nw, u0 >> 2, nu, xu0, xnu, b0, s0, acc, lane);
            }
            // ring slots that this item had no group for take the next one's as well
#pragma unroll
            for (int d = 0; d < D; ++d)
                if (!w || 4 * d >= nu) fill_group<TYPE>(ring[d], nw, (xu0 >> 2) + d, max(0, min(4, xnu - 4 * d)), lane);
            const float out_scale = TYPE == CHIMERE_TYPE_Q4_0 ? 0x1p45f : 0x1p49f;
            const int quad = lane >> 2, tg = lane & 3;
            if (STAGE == 1 && wk == 1) {
                // a warp owns its rows' whole sums: straight to the per-pair rows
                if (w) {
                    const int h0 = (rg * wr + rt_id) * 32 + quad;
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        if (t == 0 || two) {
#pragma unroll
                            for (int c = 0; c < 2; ++c) {
                                const int col = t * 8 + 2 * tg + c;
                                if (col < cols) {
                                    float* out = p.pair_out + (size_t)s_prow[buf][col] * p.H + h0;
#pragma unroll
                                    for (int i = 0; i < 4; ++i) {
                                        float lo, hi;
                                        unpack2(acc[i][t], lo, hi);
                                        out[8 * i] = (c ? hi : lo) * out_scale;
                                    }
                                }
                            }
                        }
                    }
                }
            } else {
                const int rb = step & 1;
                const uint32_t use = (uint32_t)(step >> 1) & 1u;
                bool ok = step < 2 || mbar_wait(&s_empty[rb], use ^ 1u);   // (the sums of two items ago have been read)
                float* q0 = red + (size_t)(rb * kMmaWarps + warp) * kMmaRedWarp + 2 * tg * kMmaRedPitch + quad;
#pragma unroll
                for (int t = 0; t < 2; ++t)
                    if (t == 0 || two) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            float lo, hi;
                            unpack2(acc[i][t], lo, hi);
                            float* q = q0 + t * 8 * kMmaRedPitch + 8 * i;
                            q[0] = lo * out_scale;
                            q[kMmaRedPitch] = hi * out_scale;
                        }
                    }
                __syncwarp();
                if (lane == 0) mbar_arrive_cta(&s_full[rb]);
                const int col = (warp - step) & (kMmaCols - 1);   // this warp's column of this item
                if (col < cols) {
                    ok = mbar_wait(&s_full[rb], use) && ok;
                    const float* all = red + (size_t)rb * kMmaWarps * kMmaRedWarp + col * kMmaRedPitch + lane;
                    const int orow = s_prow[buf][col], rows32 = s_tile[buf].x < 0 ? rows32_s : rows32_r;
                    for (int r = 0; r < wr; ++r) {
                        const int blk = rg * wr + r;
                        if (blk >= rows32) break;
                        float u = 0.0f, gt = 0.0f;
                        for (int s = 0; s < wk; ++s) {
                            u += all[(size_t)(r * wk + s) * kMmaRedWarp];
                            if (DUAL) gt += all[(size_t)((wr + r) * wk + s) * kMmaRedWarp];
                        }
                        if (STAGE == 1) {
                            p.pair_out[(size_t)orow * p.H + blk * 32 + lane] = u;
                            continue;
                        }
                        float v;
                        if (DUAL) v = silu_mul_ref(gt, u);
                        else { const float a = fmaxf(u, 0.0f); v = a * a; }
                        float sum = v;
#pragma unroll
                        for (int s = 16; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
                        float d;
                        const int8_t q = q8_1_warp(v, d);
                        uint8_t* out = p.inter_q8 + (size_t)orow * p.inter_stride + (size_t)blk * kQ81Bytes;
                        reinterpret_cast<int8_t*>(out)[4 + lane] = q;
                        p.out_soa_q[(size_t)orow * p.out_soa_q_stride + (size_t)blk * 32 + lane] = q;
                        if (lane == 0) {
                            const __half dh = __float2half(d);
                            *reinterpret_cast<__half2*>(out) = __halves2half2(dh, __float2half(sum));
                            p.out_soa_d[(size_t)orow * p.out_soa_d_stride + blk] = __half2float(dh);
                        }
                    }
                }
                if (!ok && lane == 0 && p.status) atomicOr(p.status, kStatusWaitTimeout);
                __syncwarp();
                if (lane == 0) mbar_arrive_cta(&s_empty[rb]);
            }
            w = nw;
            ++rg;
        }
        if (!next_tile) break;
        buf ^= 1;
        rg = 0;
        slice(buf, u0, nu);
    }
}

// ------------------------------------------------------------------ launchers --------------
static bool mma_geom(const GemvParams& p, int stage, bool dual, MmaGeom& g, size_t& smem) {
    const bool sh = p.nrows_shared > 0;
    const int wk = stage == 0 ? tiled_gate_up_geom(p.type_routed, p.type_shared, p.H, sh).wk
                              : tiled_down_geom(p.type_routed, p.ncols_routed, p.type_shared, sh ? p.ncols_shared : p.split_cols_shared, p.T).wk;
    g.wk = wk;
    g.wr = kMmaWarps / (dual ? 2 : 1) / wk;
    g.slice_r = tiled_slice_units(p.type_routed, p.ncols_routed, wk);
    g.slice_s = sh ? tiled_slice_units(p.type_shared, p.ncols_shared, wk) : 0;
    const int ncols = p.ncols_routed > p.ncols_shared && sh ? p.ncols_routed : sh ? p.ncols_shared : p.ncols_routed;
    g.pitch = ncols + 16;
    g.nb_max = ncols / 32;
    smem = 2 * mma_tile_bytes(g.pitch, g.nb_max) + (stage == 1 && wk == 1 ? 0 : (size_t)2 * kMmaWarps * kMmaRedWarp * 4);
    return smem <= 222 * 1024;
}

// Whether these kernels take a layer (both stages): one packed type per stage, planes and weights on 16-byte boundaries.
bool mma_tiles_run(const GemvParams& gu, const GemvParams& d) {
    auto ok = [](int t) { return t == CHIMERE_TYPE_Q4_0 || t == CHIMERE_TYPE_IQ3_S; };
    const bool sh = d.nrows_shared > 0;
    if (!ok(gu.type_routed) || !ok(d.type_routed) || (sh && (gu.type_shared != gu.type_routed || d.type_shared != d.type_routed))) return false;
    const uintptr_t ptrs = (uintptr_t)gu.w_a | (uintptr_t)gu.w_b | (uintptr_t)gu.sh_a | (uintptr_t)gu.sh_b | (uintptr_t)gu.stride_a | (uintptr_t)gu.stride_b |
                           (uintptr_t)gu.in_soa_q | (uintptr_t)gu.in_soa_q_stride | (uintptr_t)d.w_a | (uintptr_t)d.sh_a | (uintptr_t)d.stride_a |
                           (uintptr_t)d.in_soa_q | (uintptr_t)d.in_soa_q_stride;
    if (ptrs & 15) return false;
    MmaGeom g;
    size_t smem;
    return mma_geom(gu, 0, gu.act == CHIMERE_ACT_SWIGLU, g, smem) && mma_geom(d, 1, false, g, smem);
}

template <int TYPE, int STAGE, bool DUAL, int D>
static cudaError_t launch_mma(const GemvParams& p, const int32_t* offsets, int E, cudaStream_t stream) {
    MmaGeom g;
    size_t smem;
    if (!mma_geom(p, STAGE, DUAL, g, smem)) return cudaErrorInvalidValue;
    static bool attr_done[64] = {};
    const cudaError_t e = max_smem_once(mma_tile_kernel<TYPE, STAGE, DUAL, D>, 222 * 1024, attr_done);
    if (e != cudaSuccess) return e;
    return launch_pdl(mma_tile_kernel<TYPE, STAGE, DUAL, D>, dim3(sm_count()), kMmaThreads, smem, stream, p, offsets, E, g);
}
cudaError_t launch_mma_gate_up(const GemvParams& p, const int32_t* offsets, int E, cudaStream_t stream) {
    const bool dual = p.act == CHIMERE_ACT_SWIGLU;
    if (p.type_routed == CHIMERE_TYPE_IQ3_S)
        return dual ? launch_mma<CHIMERE_TYPE_IQ3_S, 0, true, 1>(p, offsets, E, stream) : launch_mma<CHIMERE_TYPE_IQ3_S, 0, false, 1>(p, offsets, E, stream);
    return dual ? launch_mma<CHIMERE_TYPE_Q4_0, 0, true, 1>(p, offsets, E, stream) : launch_mma<CHIMERE_TYPE_Q4_0, 0, false, 1>(p, offsets, E, stream);
}
cudaError_t launch_mma_down(const GemvParams& p, const int32_t* offsets, int E, cudaStream_t stream) {
    return p.type_routed == CHIMERE_TYPE_IQ3_S ? launch_mma<CHIMERE_TYPE_IQ3_S, 1, false, 1>(p, offsets, E, stream)
                                               : launch_mma<CHIMERE_TYPE_Q4_0, 1, false, 1>(p, offsets, E, stream);
}

}  // namespace chimere
