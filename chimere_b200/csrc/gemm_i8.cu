// gemm_i8.cu -- grouped block-scaled int8 GEMM on the 5th-generation tensor cores (tcgen05, sm_100a): the products of
// every batch whose experts hold more than a token or two.
//
// Math per output element:   D[row][tok] = sum over 32-wide blocks b of
//                            sa[row][b] * sb[tok][b] * (sum_i A[row][32b+i] * B[tok][32b+i])
// i.e. exactly the per-block integer dot of the ggml Q8_0 x Q8_1 / Q4_0 x Q8_1 / IQ3_S x Q8_1 kernels
// (chimere-server/src/kernels/gemv_q8_0.rs:230-255, chimere-server/kernels/chimere_kernels.cu:788-862),
// kept as an exact int32 per block and scaled in fp32 -- the integer results are bit-identical to the
// GEMV path; only the order of the fp32 operations differs.
//
// 4-bit weights are read in the tiled32 form the GEMV kernels use (tiled.cuh), so there is one copy of them: they travel
// packed, and two expander warps turn them into int8 on the way (16 * code for Q4_0, 8 * (2 * code + 1) for IQ3_S, the
// factor taken out of the scale).  Q8_0 weights come from a copy in the MMA's own order (mma128 tiles), because their
// tiled32 pieces would have to be copied 512 bytes at a time and a copy costs the issuing warp about 50 cycles.  Token tiles hold up to 128 pairs of one expert in the operand order (gather_tiles_kernel); a tile is
// 16, 32, 64 or 128 columns wide, whatever its pairs need.
//
// CTA = 24 warps, persistent (one CTA per SM), output tiles (128 weight rows x one token tile) from an atomic counter:
//   warp 0      takes the next tile, publishes it through a small ring, and feeds the operand rings with cp.async.bulk
//               (ring 1: packed weights and scales, token block; ring 2: the MMA's A operand);
//   warp 1      owns TMEM (512 columns) and issues the MMAs, one block = one int32 accumulator, several blocks per slot;
//   warps 2..3  expand packed weights and their scales;
//   warps 4..7  take a finished tile's sums from the exchange buffer and store it (activation and Q8_1 step, or pair rows);
//   warps 8..23 read the accumulators back (four warps per TMEM lane quarter), scale and add into fp32 registers
//               (thread = weight row), and leave a tile's sums in the exchange buffer.
// What bounds it.  Wide tiles: the read-back -- every value of every block passes through two fp32 multiply-adds on the
// CUDA cores against 32 on the tensor pipe.  The int32 -> float conversion costs nothing: each accumulator starts from
// +524288 (a constant MMA, (-128) * (-128) * 32, in front of the real one; |dot| <= 32 * 127 * 128 < 524288), so its bits are
// a positive denormal float, value * 2^-149, and the first multiply-add takes the offset and the power of two out again
// exactly (probe: 715 cycles per 128 x 128 x 32 block with an integer add per value, 597 with the constant MMA).  The
// three-operand f32x2 multiply-adds themselves take 3.2 cycles per warp (two operand pairs of the three fresh: register ports),
// i.e. 410 of those cycles.  Narrow tiles: the weight bytes, and what a stage costs its warps however few columns it has
// (an MMA takes 46 cycles at least, a commit another hundred; the read-back's shares are dealt stage by stage).
// The same tiles on the warp-level MMA, sums in registers, two CTAs of eight warps: 8192 tokens 1888 -> 2080 us, 256 wide 371 -> 437: too few
// warps to cover the way from an MMA to its multiply-adds.
// All waits are bounded; a wait that runs out raises a status bit, nothing blocks for good, and the CTA still
// frees its TMEM.
#include "common.cuh"
#include "kernels.h"
#include "tiled.cuh"

namespace chimere {

constexpr int kG_MmaTile = 4096 + 512;       // operand of one block: 128 rows x 32 int8 in the MMA's order, then 128 f32 scales
constexpr int kG_StageUnits = 4;             // 32-wide blocks per ring stage
constexpr int kG_RawBytes = 9216;            // packed weights of a stage: 4 row tiles x 4 units x 576 (Q4_0, the largest)
constexpr int kG_ASlot = kOperandMinStage, kG_ASlots = 3;   // ring 2: the A operand [4][kG_MmaTile], then (kTypeOperandMin) [4][128] minimums
constexpr int kG_RingSlotWide = kG_RawBytes + kG_StageUnits * 128 * 40, kG_RingSlotsWide = 3;
constexpr int kG_RingSlotSlim = kG_RawBytes + kG_StageUnits * 32 * 40, kG_RingSlotsSlim = 6;   // tiles of up to 32 columns
constexpr int kG_RingBytes = kG_RingSlotWide * kG_RingSlotsWide;
static_assert(kG_RingSlotSlim * kG_RingSlotsSlim <= kG_RingBytes, "both ring geometries share one area");
static_assert(kG_RingSlotsWide == kG_ASlots && kG_RingSlotsSlim == 2 * kG_ASlots, "an A slot's last user is found from the ring-1 slot of that stage");
constexpr int kG_ConstBytes = 4096;          // operand of the constant MMA
constexpr int kG_XchFloats = 128 * 128;      // exchange buffer [K share][column][128 rows]: 1 x 128, 2 x 64 or 4 x 32 columns
constexpr int kG_ExpWarps = 2, kG_EpiWarps = 4, kG_RbWarps = 16, kG_SlimExpWarps = 8;
constexpr int kG_FirstEpi = 4, kG_FirstRb = 8;
constexpr int kG_Threads = 32 * (kG_FirstRb + kG_RbWarps);
// Registers: the launch gives every thread 80; the read-back warps take 88 (512 x 88) and leave 64 to the others (256 x 64).
// (With 80 for all the read-back spills inside its loop, 1150 cycles per block instead of 700; with 96 / 48 the expanders do: 520 us
// for the Nemotron-H-style layer's 256 tokens instead of 450.)
constexpr int kG_RegsRb = 88, kG_RegsAux = 64;
static_assert(kG_RbWarps * kG_RegsRb + kG_FirstRb * kG_RegsAux == (kG_RbWarps + kG_FirstRb) * 80, "register shares add up to the launch's total");
constexpr int kG_TmemCols = 512, kG_TmemSlots = 8;
constexpr int kG_Sched = 4;                  // tile indices in flight between the scheduler and the other warps
constexpr size_t kG_Smem = 1024 + kG_ConstBytes + (size_t)kG_RingBytes + kG_ASlots * kG_ASlot + kG_XchFloats * 4;

__device__ __forceinline__ uint64_t smem_desc_kmajor(uint32_t saddr, uint32_t lbo) {
    // start address (>>4) | leading (K) byte offset (>>4) << 16 | stride (8-row group) byte offset 128 (>>4) << 32 | version 1 << 46
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(128u >> 4) << 32) | (1ull << 46);
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// One lane of a converged warp.  The single-thread roles keep their whole warp together and let the elected lane issue:
// their state is then the same in every lane and stays in uniform registers, which the MMA and copy instructions read.
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}
__device__ __forceinline__ int uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ const uint8_t* uniform(const uint8_t* v) { return (const uint8_t*)__shfl_sync(0xffffffffu, (unsigned long long)v, 0); }
__device__ __forceinline__ void tc_mma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u) : "memory");
}
// TMEM -> registers, thread = lane (row), N consecutive 32-bit columns; no wait: tc_wait_ld() before the values are used
template <int N> __device__ __forceinline__ void tc_ld_nowait(uint32_t taddr, int (&v)[N]);
template <> __device__ __forceinline__ void tc_ld_nowait<32>(uint32_t taddr, int (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
          "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
          "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr) : "memory");
}
template <> __device__ __forceinline__ void tc_ld_nowait<16>(uint32_t taddr, int (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr) : "memory");
}
template <> __device__ __forceinline__ void tc_ld_nowait<8>(uint32_t taddr, int (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// two 64-bit words (four floats) from a 32-bit shared address, the same for every lane
__device__ __forceinline__ void lds_2x64(uint32_t a, uint64_t& x, uint64_t& y) { asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"(a)); }
__device__ __forceinline__ float lds_f32(uint32_t a) { float v; asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a)); return v; }
__device__ __forceinline__ void sts128(uint32_t a, uint4 v) { asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory"); }
__device__ __forceinline__ void sts_f32(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }

// The powers of two of the read-back: an accumulator's float reading is (dot + 2^19) * 2^-149.  The first multiply-add takes
// scale * 2^100 and the offset -2^19 * 2^-149 * (scale * 2^100), and the finished sums are multiplied by 2^49.  All exact;
// the intermediate sums stay far inside fp32's normal range for any f16 scales.
constexpr uint32_t kRowScaleBits = 0x71800000u;      // 2^100
constexpr uint32_t kOffsetBits = 0xB0800000u;        // -2^-30 = -2^19 * 2^-149 * 2^100
constexpr uint32_t kSumScaleBits = 0x58000000u;      // 2^49

struct GemmShared {
    uint64_t full1[kG_RingSlotsSlim];                // ring 1: a stage's bytes have landed (kTypeOperand: those of ring 2 as well)
    uint64_t empty1[kG_RingSlotsSlim];               // ... the stage has been read back, and both its slots are free: one arrival of every
                                                     // read-back warp, whatever its part in the tile
    uint64_t xfull2[kG_ASlots];                      // ring 2: operand and scales expanded
    uint64_t tfull[kG_TmemSlots], tempty[kG_TmemSlots];   // accumulators of a slot complete / read back (tempty: wide tiles only)
    uint64_t sfull[kG_Sched], sempty[kG_Sched];      // a tile index has been published / taken by every other warp
    uint64_t xfull, xempty;                          // a tile's sums are in the exchange buffer / have been stored
    int sched[kG_Sched];
    uint32_t tmem_base;
    int failed;
};

// One output tile: 128 weight rows (row tile rt of an expert's matrix) x the columns of a token tile.
struct GemmWork {
    const uint8_t* b;            // token tile: [block][npad * 36 bytes]
    int nb;                      // 32-wide blocks of K
    int n_valid, npad;           // token columns / as laid out (16, 32, 64 or 128)
    int expert, shared, rt, start, col16;
    int aux0, aux1;
};
constexpr int kWorkOk = 0, kWorkSkip = 1, kWorkEnd = 2;
// Kernel instances.  kMin: the tiles with minimums (Q4_K / Q5_K shared expert) and no others.  kOrdered: the decode entry's tiles, whose
// sums are bit for bit the GEMV kernels' (readback_ordered): packed weights, tiles of up to 64 columns.
constexpr int kPlain = 0, kMin = 1, kOrdered = 2;
struct RowTiles { const uint8_t* src0; const uint8_t* src1; int tile_bytes, n0, n1; };   // the 32-row tiles of a GemmWork (see produce_tile)

// Position in the two operand rings; every role walks the same sequence.  Ring 1 has two geometries (slots for tiles of
// more than 32 columns, and more, smaller ones); on a change the producer lets the ring run empty first.
struct RingPos {
    int r = 0, e = 0, slim = 0;
    uint32_t ph1 = 0, ph2 = 0;
    __device__ __forceinline__ int slots1() const { return slim ? kG_RingSlotsSlim : kG_RingSlotsWide; }
    __device__ __forceinline__ uint32_t slot1_off() const { return (uint32_t)r * (slim ? kG_RingSlotSlim : kG_RingSlotWide); }
    __device__ __forceinline__ void geometry(int s) { if (s != slim) { slim = s; r = 0; } }
    __device__ __forceinline__ uint32_t par1() const { return (ph1 >> r) & 1u; }
    __device__ __forceinline__ uint32_t par2() const { return (ph2 >> e) & 1u; }
    // the ring-1 slot of the stage that used A slot e before (three stages ago), and the parity its release completes
    __device__ __forceinline__ int lag() const { return slim ? (r >= kG_ASlots ? r - kG_ASlots : r + kG_ASlots) : r; }
    __device__ __forceinline__ uint32_t released(int slot) const { return ((ph1 >> slot) & 1u) ^ 1u; }
    __device__ __forceinline__ void next(bool expanded) {
        ph1 ^= 1u << r;
        if (expanded) ph2 ^= 1u << e;
        r = r + 1 == slots1() ? 0 : r + 1;
        e = e + 1 == kG_ASlots ? 0 : e + 1;
    }
};
// (All waits are on parities.  Who waits on a barrier has to be someone without whom it cannot go two phases on: a stage is released by
// all 16 read-back warps, each of which has seen its accumulators complete or has expanded it; MMA and expander warps are held by what they
// feed; warps 2..3, which sit out some tiles, come back to drained rings.)
// TMEM slots of a tile of npad columns (512 columns in all): two blocks per slot in a 128-column tile, else a whole stage.
struct TmemPos {
    int slot = 0, npad = 0, nslots = 0;
    uint32_t ph = 0, ph_empty = 0;   // (ph_empty: the MMA warp's, of the slots that wait for their read-back)
    __device__ __forceinline__ uint32_t par() const { return (ph >> slot) & 1u; }
    __device__ __forceinline__ void next() { ph ^= 1u << slot; slot = slot + 1 == nslots ? 0 : slot + 1; }
};
__host__ __device__ constexpr int blocks_per_slot(int npad) { return npad == 128 ? 2 : 4; }

// arrival of one thread for `n` of a barrier's count
__device__ __forceinline__ void mbar_arrive_n(uint64_t* bar, uint32_t n) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(n) : "memory");
}
// A wait ran out: noted here, reported by the CTA's last step.
__device__ __forceinline__ void gemm_timeout(GemmShared& sh) { sh.failed = 1; }

// ------------------------------------------------------------------ roles ----
// First unit of stage s.  IQ3_S tiles keep a super-block's scales behind its eight units, so its second half is taken first
// (one copy brings both) and the expanders keep the scales for the first half; kOrdered takes the units as they come and the
// scales with a copy of their own.
template <int MODE>
__device__ __forceinline__ int stage_unit(int type, int s) { return kG_StageUnits * (MODE != kOrdered && type == CHIMERE_TYPE_IQ3_S ? s ^ 1 : s); }

// Warp 0: copies of one tile, a few pieces per stage, all issued by the elected lane (a copy costs its warp about 50 cycles).
template <class Policy, int MODE, class Params>
__device__ __forceinline__ bool produce_tile(const Params& p, const GemmWork& w, GemmShared& sh, uint8_t* ring1, uint8_t* ring2, RingPos& pos, int lane) {
    const int type = uniform(Policy::type(p, w)), nb = uniform(w.nb), npad = uniform(w.npad);
    const bool operand = MODE != kOrdered && type >= kTypeOperand;
    const int slim = npad <= 32;
    if (slim != pos.slim) {   // the other slot geometry: every slot of the old one has to be empty first
        for (int r = 0; r < pos.slots1(); ++r)
            if (!mbar_wait(&sh.empty1[r], pos.released(r))) { gemm_timeout(sh); return false; }
        pos.geometry(slim);
    }
    // four row tiles: two at src0, two at src1 (neighbours tile_bytes apart), n0 and n1 of them there
    const RowTiles rt = Policy::rows(p, w);
    const uint8_t* src0 = uniform(rt.src0);
    const uint8_t* src1 = uniform(rt.src1);
    const uint8_t* bsrc = uniform(w.b);
    const uint32_t tile_bytes = (uint32_t)uniform(rt.tile_bytes), n0 = (uint32_t)uniform(rt.n0), n1 = (uint32_t)uniform(rt.n1);
    const int nstages = (nb + kG_StageUnits - 1) / kG_StageUnits;
    for (int s = 0; s < nstages; ++s) {
        const int u0 = stage_unit<MODE>(type, s), nu = min(kG_StageUnits, nb - u0);
        uint64_t* bar = &sh.full1[pos.r];
        bool ok = mbar_wait(&sh.empty1[pos.r], pos.released(pos.r));
        if (ok && operand) ok = mbar_wait(&sh.empty1[pos.lag()], pos.released(pos.lag()));
        if (!ok) { gemm_timeout(sh); return false; }
        uint8_t* raw = ring1 + pos.slot1_off();
        // a token block: 32 values and a scale per column, beside weights with minimums the column's sum as well (by stages)
        const uint32_t bcol = type == kTypeOperandMin ? 40u : 36u, bbytes = (uint32_t)(nu * npad) * bcol;
        // 4-bit types: bytes of one row tile, and where they start in it
        const uint32_t piece = type == CHIMERE_TYPE_Q4_0 ? (uint32_t)nu * 576u : (s & 1) || MODE == kOrdered ? 2048u : 2240u;
        const bool scales = MODE == kOrdered && type == CHIMERE_TYPE_IQ3_S && !(s & 1);   // (behind the super-block's units, 192 bytes)
        const uint32_t off = type == CHIMERE_TYPE_Q4_0 ? (uint32_t)u0 * 576u : (uint32_t)(u0 >> 3) * 4288u + (uint32_t)(u0 & 4) * 512u;
        if (elect_one()) {
            if (operand) {
                const uint32_t abytes = (uint32_t)nu * (type == kTypeOperand ? kG_MmaTile : kOperandMinStage / kG_StageUnits);
                mbar_expect_tx(bar, abytes + bbytes);
                bulk_g2s(ring2 + (uint32_t)pos.e * kG_ASlot, src0 + (size_t)u0 * (type == kTypeOperand ? kG_MmaTile : kOperandMinStage / kG_StageUnits), abytes, bar);
            } else {
                mbar_expect_tx(bar, (n0 + n1) * (piece + (scales ? 192u : 0u)) + bbytes);
                const uint8_t* a = src0 + off;
                const uint8_t* b = src1 + off;
                bulk_g2s(raw, a, piece, bar);
                if (n0 > 1) bulk_g2s(raw + kG_RawBytes / 4, a + tile_bytes, piece, bar);
                if (n1 > 0) bulk_g2s(raw + kG_RawBytes / 2, b, piece, bar);
                if (n1 > 1) bulk_g2s(raw + 3 * (kG_RawBytes / 4), b + tile_bytes, piece, bar);
                if (scales) {
                    bulk_g2s(raw + 2048, a + 4096, 192u, bar);
                    if (n0 > 1) bulk_g2s(raw + kG_RawBytes / 4 + 2048, a + tile_bytes + 4096, 192u, bar);
                    if (n1 > 0) bulk_g2s(raw + kG_RawBytes / 2 + 2048, b + 4096, 192u, bar);
                    if (n1 > 1) bulk_g2s(raw + 3 * (kG_RawBytes / 4) + 2048, b + tile_bytes + 4096, 192u, bar);
                }
            }
            bulk_g2s(raw + kG_RawBytes, bsrc + (size_t)u0 * (npad * bcol), bbytes, bar);
        }
        __syncwarp();
        pos.next(!operand);
    }
    return true;
}

// Packed 4-bit units -> int8 operand rows.  A unit's 16 bytes per row hold elements 0..15 in the low nibbles (code + 8) and
// 16..31 in the high ones (two's complement): the two halves are the row's 16 bytes of the operand's two K halves.
// Warp x expands row tiles x and x + 2; all loads of a stage go out first (the compiler keeps the order of the
// shared-memory accesses as written).
template <int TYPE>
__device__ __forceinline__ void expand_unit(const uint4& v, uint32_t dst) {
    constexpr uint32_t kOdd = TYPE == CHIMERE_TYPE_IQ3_S ? 0x08080808u : 0u;   // 8 * (2c + 1) = 16c + 8
    uint4 lo, hi;
    lo.x = ((v.x << 4) & 0xF0F0F0F0u) ^ (0x80808080u | kOdd); hi.x = (v.x & 0xF0F0F0F0u) | kOdd;
    lo.y = ((v.y << 4) & 0xF0F0F0F0u) ^ (0x80808080u | kOdd); hi.y = (v.y & 0xF0F0F0F0u) | kOdd;
    lo.z = ((v.z << 4) & 0xF0F0F0F0u) ^ (0x80808080u | kOdd); hi.z = (v.z & 0xF0F0F0F0u) | kOdd;
    lo.w = ((v.w << 4) & 0xF0F0F0F0u) ^ (0x80808080u | kOdd); hi.w = (v.w & 0xF0F0F0F0u) | kOdd;
    sts128(dst, lo);
    sts128(dst + 2048, hi);
}
constexpr uint32_t kRawTile = kG_RawBytes / 4;   // a row tile's packed units in a ring slot
template <int TYPE> __host__ __device__ constexpr uint32_t raw_unit() { return TYPE == CHIMERE_TYPE_IQ3_S ? 512 : 576; }
template <int TYPE>
__device__ __forceinline__ void expand_units(uint32_t raw, uint32_t a, int x, int lane) {
    const uint32_t src = raw + (uint32_t)x * kRawTile + lane * 16, dst = a + (uint32_t)x * 512 + lane * 16;
    uint4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = lds128(src + (i & 1) * 2 * kRawTile + (i >> 1) * raw_unit<TYPE>());   // (units past nu: bytes nobody uses)
#pragma unroll
    for (int i = 0; i < 8; ++i) expand_unit<TYPE>(v[i], dst + (i >> 1) * kG_MmaTile + (i & 1) * 1024);
}

// The word beside an expanded IQ3_S row of a unit: d * (1 + 2 * sub-scale) / 8 (exact in f32), or (kOrdered, which multiplies by the two
// factors where the GEMV kernels do) f16 d in the upper half and 1 + 2 * sub-scale in the lower.
template <int MODE>
__device__ __forceinline__ uint32_t iq3s_word(uint32_t d16, uint32_t sub) {
    return MODE == kOrdered ? (d16 << 16) | (1u + 2u * sub) : __float_as_uint(h2f(d16) * 0.125f * (float)(1u + 2u * sub));
}
__device__ __forceinline__ void sts_u32(uint32_t a, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }

// Whether warps 2..3 expand a tile's weights: not those in operand order, and in slim tiles half of the read-back warps do it.
template <int MODE>
__device__ __forceinline__ bool warps23_expand(int type, bool slim) { return (MODE == kOrdered || type < kTypeOperand) && !slim; }

// Warps 2..3: warp x takes row tiles x and x + 2 of every stage.
template <class Policy, int MODE, class Params>
__device__ __forceinline__ bool expand_tile(const Params& p, const GemmWork& w, GemmShared& sh, uint32_t ring1, uint32_t ring2, RingPos& pos, int x, int lane) {
    const int type = uniform(Policy::type(p, w)), nb = uniform(w.nb);
    const bool slim = uniform(w.npad) <= 32;
    pos.geometry(slim);
    const int nstages = (nb + kG_StageUnits - 1) / kG_StageUnits;
    if (!warps23_expand<MODE>(type, slim)) {   // nothing to do but keep step; no waits: nothing holds the rings back for these warps here
        for (int s = 0; s < nstages; ++s) pos.next(MODE == kOrdered || type < kTypeOperand);
        return true;
    }
    uint32_t d3[2] = {0u, 0u}, sc3[2] = {0u, 0u};   // IQ3_S: this lane's rows' scales of the super-block, kept over its two stages
    for (int s = 0; s < nstages; ++s) {
        const int u0 = stage_unit<MODE>(type, s);
        if (!mbar_wait(&sh.full1[pos.r], pos.par1()) || !mbar_wait(&sh.empty1[pos.lag()], pos.released(pos.lag()))) { gemm_timeout(sh); return false; }
        const uint32_t raw = ring1 + pos.slot1_off(), a = ring2 + (uint32_t)pos.e * kG_ASlot;
        const uint32_t rec = a + 4096 + (x * 32 + lane) * 4;   // [unit] kG_MmaTile apart, row tile x + 2: 256 bytes further
        if (type == CHIMERE_TYPE_Q4_0) {
            expand_units<CHIMERE_TYPE_Q4_0>(raw, a, x, lane);
            uint32_t d[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) d[i] = lds16(raw + (x + 2 * (i & 1)) * (kG_RawBytes / 4) + (i >> 1) * 576 + 512 + lane * 2);
#pragma unroll
            for (int i = 0; i < 8; ++i) sts_f32(rec + (i >> 1) * kG_MmaTile + (i & 1) * 256, h2f(d[i]) * 0.0625f);
        } else {
            expand_units<CHIMERE_TYPE_IQ3_S>(raw, a, x, lane);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (!(s & 1)) {   // the scales came behind these units
                    const uint32_t t = raw + (x + 2 * h) * (kG_RawBytes / 4) + 2048;
                    d3[h] = lds16(t + lane * 2);
                    sc3[h] = lds32(t + 64 + lane * 4);
                }
                const uint32_t sc = sc3[h] >> (4 * (u0 & 4));
#pragma unroll
                for (int u = 0; u < 4; ++u) sts_u32(rec + u * kG_MmaTile + h * 256, iq3s_word<MODE>(d3[h], (sc >> (4 * u)) & 15u));
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the MMAs read what ordinary stores wrote
        __syncwarp();
        if (lane == 0) mbar_arrive_n(&sh.xfull2[pos.e], kG_SlimExpWarps / kG_ExpWarps);
        pos.next(true);
    }
    return true;
}

// Warp 1: the MMAs of one tile, issued by its elected lane.  A slim tile's TMEM slots need no barrier of their own: there are
// more of them than A slots, and an A slot is refilled only after its stage has been read back.  Everything a block's MMA
// needs is a constant away from the stage's values: with a slim tile the warp has about 400 cycles per stage, of which the
// four MMAs and the commit take 360.
template <class Policy, int MODE, int NPAD, class Params>
__device__ __forceinline__ bool mma_tile(const Params& p, const GemmWork& w, GemmShared& sh, uint32_t cst, uint32_t ring1, uint32_t ring2, uint32_t tmem,
                                         RingPos& pos, TmemPos& tp, int lane) {
    constexpr int kBps = blocks_per_slot(NPAD);
    constexpr bool kWide = NPAD == 128, kHandshake = NPAD >= 64;
    // D format S32 (2 << 4), A and B signed int8 (1 << 7, 1 << 10), both K-major, N (>> 3 at bit 17), M = 128 (>> 4 at bit 24)
    constexpr uint32_t kIdesc = (2u << 4) | (1u << 7) | (1u << 10) | (((uint32_t)NPAD >> 3) << 17) | ((128u >> 4) << 24);
    const bool expanded = MODE == kOrdered || uniform(Policy::type(p, w)) < kTypeOperand;
    const int nb = uniform(w.nb);
    if (NPAD != tp.npad) {   // another width lays the accumulators out differently: everything has to be read back first
        for (int r = 0; r < pos.slots1(); ++r)
            if (!mbar_wait(&sh.empty1[r], pos.released(r))) { gemm_timeout(sh); return false; }
        tp.npad = NPAD; tp.slot = 0; tp.nslots = kG_TmemCols / (kBps * NPAD);
    }
    pos.geometry(NPAD <= 32);
    const uint64_t ca = smem_desc_kmajor(cst, 2048), cb = smem_desc_kmajor(cst, NPAD * 16);
    const uint64_t a_base = smem_desc_kmajor(ring2, 2048), b_base = smem_desc_kmajor(ring1 + kG_RawBytes, NPAD * 16);
    auto block = [&](uint64_t a, uint64_t b, uint32_t d, int j) {
        d += (uint32_t)((j % kBps) * NPAD);
        if (kWide) tc_mma_i8(d, ca, cb, kIdesc, 0u);
        tc_mma_i8(d, a + (uint32_t)(j * (kG_MmaTile >> 4)), b + (uint32_t)(j * ((NPAD * 36) >> 4)), kIdesc, kWide ? 1u : 0u);
    };
    for (int b0 = 0; b0 < nb; b0 += kG_StageUnits) {
        const int nu = min(kG_StageUnits, nb - b0);
        if (!(expanded ? mbar_wait(&sh.xfull2[pos.e], pos.par2()) : mbar_wait(&sh.full1[pos.r], pos.par1()))) { gemm_timeout(sh); return false; }
        const uint64_t a = a_base + (uint32_t)pos.e * (kG_ASlot >> 4), b = b_base + (pos.slot1_off() >> 4);
#pragma unroll
        for (int j0 = 0; j0 < kG_StageUnits; j0 += kBps) {
            if (j0 >= nu) break;
            if (kHandshake) {
                if (!mbar_wait(&sh.tempty[tp.slot], ((tp.ph_empty >> tp.slot) & 1u) ^ 1u)) { gemm_timeout(sh); return false; }
                tp.ph_empty ^= 1u << tp.slot;
            }
            tc_fence_after();
            const uint32_t d = tmem + (uint32_t)(tp.slot * (kBps * NPAD));
            if (elect_one()) {
                if (nu == kG_StageUnits) {
#pragma unroll
                    for (int j = 0; j < kBps; ++j) block(a, b, d, j0 + j);
                } else {
                    for (int j = j0; j < min(nu, j0 + kBps); ++j) block(a, b, d, j);
                }
                tc_commit(&sh.tfull[tp.slot]);   // (also tells the read-back warps that the operands have been read)
            }
            __syncwarp();
            tp.next();
        }
        pos.next(expanded);
    }
    return true;
}

// W accumulator columns of this thread's row: acc[c] += (dot * sa) * sb[c] with dot * sa = fma(reading, sa, offset * sa),
// rounded once like a plain product.  sb: shared address of the first column's token scale.
// ANY_SCALE: scales may be any f32 (2^100 times one above 2^28 is infinite), so the exact dot comes first, without a power of two.
template <int W, uint32_t kBias, bool ANY_SCALE>
__device__ __forceinline__ void block_values(const int (&v)[W], float sa, uint32_t sb, uint64_t* acc2) {
    if (ANY_SCALE) {
        const uint64_t r2 = pack2(kRowScaleBits, kRowScaleBits), o2 = pack2(kOffsetBits, kOffsetBits), p2 = pack2(kSumScaleBits, kSumScaleBits), a2 = pack2f(sa, sa);
#pragma unroll
        for (int g = 0; g < W / 4; ++g) {
            uint64_t s[2];
            lds_2x64(sb + 16u * g, s[0], s[1]);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint64_t t = mul2(fma2(pack2((uint32_t)v[4 * g + 2 * i] + kBias, (uint32_t)v[4 * g + 2 * i + 1] + kBias), r2, o2), p2);
                acc2[2 * g + i] = fma2(mul2(t, a2), s[i], acc2[2 * g + i]);
            }
        }
        return;
    }
    const float sr = sa * __uint_as_float(kRowScaleBits), c = sa * __uint_as_float(kOffsetBits);
    const uint64_t sa2 = pack2f(sr, sr);
    const uint64_t c2 = pack2f(c, c);
#pragma unroll
    for (int g = 0; g < W / 4; ++g) {
        uint64_t s01, s23;
        lds_2x64(sb + 16u * g, s01, s23);
        const uint64_t u01 = fma2(pack2((uint32_t)v[4 * g + 0] + kBias, (uint32_t)v[4 * g + 1] + kBias), sa2, c2);
        const uint64_t u23 = fma2(pack2((uint32_t)v[4 * g + 2] + kBias, (uint32_t)v[4 * g + 3] + kBias), sa2, c2);
        acc2[2 * g + 0] = fma2(u01, s01, acc2[2 * g + 0]);
        acc2[2 * g + 1] = fma2(u23, s23, acc2[2 * g + 1]);
    }
}

// The read-back of one tile by one warp: column group colg of W columns; in tiles of up to 64 columns the warps of a column
// group also share the stages among them (KG shares, stage s to share s % KG), so that a warp has that much longer for the
// latency of one stage (barrier, TMEM load, scales: about a thousand cycles).
template <int COLG, int KG, int W, bool ANY_SCALE>
__device__ __forceinline__ bool readback_tile(GemmShared& sh, uint32_t ring1, uint32_t ring2, uint32_t tmem, int32_t* status, int nb, bool expanded, int q,
                                              int part, int lane, RingPos& pos, TmemPos& tp, uint64_t* acc2) {
    constexpr int kPad = COLG * W, kBps = blocks_per_slot(kPad);
    constexpr bool kHandshake = kPad >= 64;
    const int colg = part % COLG, kg = part / COLG;
    if (tp.npad != kPad) { tp.npad = kPad; tp.slot = 0; tp.nslots = kG_TmemCols / (kBps * kPad); }
    const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(colg * W);
    const uint32_t rec0 = ring2 + 4096 + (uint32_t)(q * 32 + lane) * 4u;
    const uint32_t sb0 = ring1 + kG_RawBytes + kPad * 32 + colg * (W * 4);
    int share = 0;
    for (int b0 = 0; b0 < nb; b0 += kG_StageUnits) {
        const int nu = min(kG_StageUnits, nb - b0);
        if (KG > 1 && share != kg) {   // another share's stage: seen and released like its own, so that no warp is ever two phases behind a barrier
            if (!mbar_wait(&sh.tfull[tp.slot], tp.par())) { gemm_timeout(sh); return false; }
            if (kHandshake && lane == 0) mbar_arrive_cta(&sh.tempty[tp.slot]);
            tp.next();
        } else {
            const uint32_t rec = rec0 + (uint32_t)pos.e * kG_ASlot, sb = sb0 + pos.slot1_off();
#pragma unroll
            for (int j0 = 0; j0 < kG_StageUnits; j0 += kBps) {
                if (j0 >= nu) break;
                if (!mbar_wait(&sh.tfull[tp.slot], tp.par())) { gemm_timeout(sh); return false; }
                tc_fence_after();
                const uint32_t t0 = trow + (uint32_t)(tp.slot * (kBps * kPad));
                const int cnt = min(kBps, nu - j0);
#pragma unroll
                for (int i = 0; i < kBps; ++i) {
                    if (i < cnt) {
                        int v[W];
                        tc_ld_nowait<W>(t0 + (uint32_t)(i * kPad), v);
                        const float sa = lds_f32(rec + (j0 + i) * kG_MmaTile);
                        tc_wait_ld();
                        if (kHandshake && i + 1 == cnt) {   // the slot's last values are in registers: the MMAs may overwrite it
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive_cta(&sh.tempty[tp.slot]);
                        }
                        block_values<W, kPad == 128 ? 0u : 1u << 19, ANY_SCALE>(v, sa, sb + (uint32_t)((j0 + i) * (kPad * 36)), acc2);
                    }
                }
                tp.next();
            }
            if (!kHandshake) tc_fence_before();
            __syncwarp();
        }
        if (lane == 0) mbar_arrive_cta(&sh.empty1[pos.r]);
        if (KG > 1) share = share + 1 == KG ? 0 : share + 1;
        pos.next(expanded);
    }
    return true;
}

// The read-back of one tile of packed weights by one warp, W of its columns and every stage, bit for bit what the GEMV kernels compute
// for a token (gemv_tiled.cu), so that a token of a decode batch does not depend on how many others chose the same expert: with the
// exact block dot t,  acc = fma(d * dx, t, acc) per block of Q4_0;  part = fma(t, dx, part) over the four blocks of a stage and
// acc = fma(d, part, acc) for IQ3_S (t with the sub-block's factor);  slices of K (`slice` stages each) added up in order.  All sums carry 2^-49: t comes out of the
// accumulator's float reading with one exact multiply-add (IQ3_S operands are 8, Q4_0 ones 16 times the weight; the Q4_0 scale in
// shared memory is d / 16).
template <int TYPE, int COLG, int W>
__device__ __forceinline__ bool readback_ordered(GemmShared& sh, uint32_t ring1, uint32_t ring2, uint32_t tmem, int32_t* status, int nb, int slice, int q,
                                                 int colg, int lane, RingPos& pos, TmemPos& tp, uint64_t (&total)[W / 2]) {
    constexpr int kPad = COLG * W;
    constexpr bool kHandshake = kPad >= 64, kGroup = TYPE == CHIMERE_TYPE_IQ3_S;
    if (tp.npad != kPad) { tp.npad = kPad; tp.slot = 0; tp.nslots = kG_TmemCols / (kG_StageUnits * kPad); }
    const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(colg * W);
    const uint32_t rec0 = ring2 + 4096 + (uint32_t)(q * 32 + lane) * 4u, sb0 = ring1 + kG_RawBytes + kPad * 32 + colg * (W * 4);
    uint64_t acc[W / 2];
#pragma unroll
    for (int i = 0; i < W / 2; ++i) acc[i] = total[i] = 0ull;
    int left = slice;
    for (int b0 = 0; b0 < nb; b0 += kG_StageUnits) {
        const int nu = min(kG_StageUnits, nb - b0);
        const uint32_t rec = rec0 + (uint32_t)pos.e * kG_ASlot, sb = sb0 + pos.slot1_off();
        if (!mbar_wait(&sh.tfull[tp.slot], tp.par())) { gemm_timeout(sh); return false; }
        tc_fence_after();
        const uint32_t t0 = trow + (uint32_t)(tp.slot * (kG_StageUnits * kPad));
        uint64_t part[W / 2];
        uint32_t word = 0;
#pragma unroll
        for (int i = 0; i < W / 2; ++i) part[i] = 0ull;
#pragma unroll
        for (int j = 0; j < kG_StageUnits; ++j) {
            if (j >= nu) break;
            int v[W];
            tc_ld_nowait<W>(t0 + (uint32_t)(j * kPad), v);
            word = lds32(rec + j * kG_MmaTile);
            // 2^100; 2^97 times the factor: the exact dot times 2^-49 (times 16 for Q4_0), and what takes the offset 2^19 out again
            const float m = kGroup ? (float)(word & 0xFFFFu) : 1.0f;
            const float kr = kGroup ? m * __uint_as_float(kRowScaleBits - (3u << 23)) : __uint_as_float(kRowScaleBits);
            const float ko = kGroup ? m * __uint_as_float(kOffsetBits - (3u << 23)) : __uint_as_float(kOffsetBits);
            const uint64_t r2 = pack2f(kr, kr), o2 = pack2f(ko, ko), d2 = pack2(word, word);
            tc_wait_ld();
            if (kHandshake && j + 1 == nu) {   // the slot's last values are in registers: the MMAs may overwrite it
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cta(&sh.tempty[tp.slot]);
            }
#pragma unroll
            for (int g = 0; g < W / 4; ++g) {
                uint64_t s[2];
                lds_2x64(sb + (uint32_t)(j * (kPad * 36)) + 16u * g, s[0], s[1]);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint64_t t = fma2(pack2((uint32_t)v[4 * g + 2 * i] + (1u << 19), (uint32_t)v[4 * g + 2 * i + 1] + (1u << 19)), r2, o2);
                    if (kGroup) part[2 * g + i] = fma2(t, s[i], part[2 * g + i]);
                    else acc[2 * g + i] = fma2(mul2(d2, s[i]), t, acc[2 * g + i]);
                }
            }
        }
        tp.next();
        if (!kHandshake) tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cta(&sh.empty1[pos.r]);
        pos.next(true);
        if (kGroup) {
            const float d = h2f(word >> 16);
            const uint64_t d2 = pack2f(d, d);
#pragma unroll
            for (int i = 0; i < W / 2; ++i) acc[i] = fma2(d2, part[i], acc[i]);
        }
        if (--left == 0 || b0 + kG_StageUnits >= nb) {   // a slice of K is complete
            left = slice;
#pragma unroll
            for (int i = 0; i < W / 2; ++i) { total[i] = add2(total[i], acc[i]); acc[i] = 0ull; }
        }
    }
    return true;
}

// The binary counter of readback_min: sum completes level after level as long as that level has a pending left half.  The first two levels'
// pending sums are in registers, the others (a thread's share of `upper`: [level - 2][4][512 threads]) in shared memory.
constexpr int kMinRegLevels = 2, kMinLevels = 5;
template <int L>
__device__ __forceinline__ void count_up(int n, uint64_t (&sum)[4], uint64_t (&st)[kMinRegLevels][4], uint64_t* upper) {
    if constexpr (L < kMinLevels) {
        uint64_t* up = upper + (L - kMinRegLevels) * 4 * (32 * kG_RbWarps);
        if ((n >> L) & 1) {
#pragma unroll
            for (int i = 0; i < 4; ++i) sum[i] = add2(L < kMinRegLevels ? st[L < kMinRegLevels ? L : 0][i] : up[i * (32 * kG_RbWarps)], sum[i]);
            count_up<L + 1>(n, sum, st, upper);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (L < kMinRegLevels) st[L < kMinRegLevels ? L : 0][i] = sum[i];
                else up[i * (32 * kG_RbWarps)] = sum[i];
            }
        }
    }
}

// A warp's sums of a tile into the exchange buffer (part = share * column groups + column group).
template <int W, bool UNSCALED = false>
__device__ __forceinline__ bool publish_sums(int32_t* status, GemmShared& sh, float* xch, int q, int part, int lane, uint32_t& xphase, const uint64_t* acc2, bool ok) {
    if (!mbar_wait(&sh.xempty, (xphase & 1u) ^ 1u)) { gemm_timeout(sh); ok = false; }   // the tile before has been stored
    ++xphase;
    float* mine = xch + part * (W * 128) + q * 32 + lane;
    const uint64_t sc2 = pack2(kSumScaleBits, kSumScaleBits);
#pragma unroll
    for (int i = 0; i < W / 2; ++i) unpack2(UNSCALED ? acc2[i] : mul2(acc2[i], sc2), mine[(2 * i) * 128], mine[(2 * i + 1) * 128]);
    __syncwarp();
    if (lane == 0) mbar_arrive_cta(&sh.xfull);
    return ok;
}

// The read-back of a tile with minimums (Q4_K / Q5_K weights), 32 columns wide, eight of them per warp, bit for bit what
// kquant_mmvq_kernel computes: a block's value is fma(-dmin * m, s, (d * d8) * float(sc * dot)), a lane's blocks (leaf of them, in
// sequence) make a leaf, and the leaves of the 32 lanes, which come in bit-reversed order (operand_min_block), go up a binary counter
// of pending sums.  The 8-bit rounding of the intermediates would show a different order of additions: these weights reach 4 sigma,
// and one step of an intermediate moves an output by up to 3 % of the outputs' rms.  leaf = nb: plain sequence.
// (Tiles with minimums have a kernel instance of their own, so that these registers do not weigh on the other tiles' loops.)
__device__ __forceinline__ bool readback_min(GemmShared& sh, uint32_t ring1, uint32_t ring2, float* xch, uint32_t tmem, int32_t* status, int nb, int leaf, int q,
                                          int part, int lane, RingPos& pos, TmemPos& tp, uint32_t& xphase) {
    constexpr int W = 8, kPad = 32;
    static_assert(kPad * 128 * 4 + (kMinLevels - kMinRegLevels) * 4 * 32 * kG_RbWarps * 8 <= kG_XchFloats * 4, "the upper levels lie behind the 32 columns of the exchange buffer");
    pos.geometry(1);
    if (tp.npad != kPad) { tp.npad = kPad; tp.slot = 0; tp.nslots = kG_TmemCols / (blocks_per_slot(kPad) * kPad); }
    const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(part * W);
    const uint32_t rec0 = ring2 + (uint32_t)(q * 32 + lane) * 4u, sb0 = ring1 + kG_RawBytes + part * (W * 4);
    uint64_t* upper = reinterpret_cast<uint64_t*>(xch + kPad * 128) + (part * 4 + q) * 32 + lane;
    uint64_t sum[W / 2], st[kMinRegLevels][W / 2];
    int in_leaf = 0, n = 0;
    bool ok = true;
    for (int b0 = 0; b0 < nb && ok; b0 += kG_StageUnits) {
        const uint32_t rec = rec0 + (uint32_t)pos.e * kG_ASlot, sb = sb0 + pos.slot1_off();
        if (!mbar_wait(&sh.tfull[tp.slot], tp.par())) { ok = false; break; }
        tc_fence_after();
        const uint32_t t0 = trow + (uint32_t)(tp.slot * (kG_StageUnits * kPad));
        // a stage's accumulators at once: one wait for the TMEM instead of four (half-layer of 777 tokens with a Q5_K shared expert 519 -> 449 us,
        // with these tiles launched behind the others instead of in front)
        int v[kG_StageUnits][W];
#pragma unroll
        for (int j = 0; j < kG_StageUnits; ++j) tc_ld_nowait<W>(t0 + (uint32_t)(j * kPad), v[j]);
        tc_wait_ld();
#pragma unroll
        for (int j = 0; j < kG_StageUnits; ++j) {
            const uint32_t ds = lds32(rec + 4096 + j * kG_MmaTile);
            const float m = lds_f32(rec + 4 * kG_MmaTile + j * 512), d = h2f(ds >> 16), sc = (float)(ds & 63u);
            const uint64_t sc2 = pack2f(sc * __uint_as_float(kRowScaleBits), sc * __uint_as_float(kRowScaleBits));
            const uint64_t c2 = pack2f(sc * __uint_as_float(kOffsetBits), sc * __uint_as_float(kOffsetBits)), d2 = pack2f(d, d), m2 = pack2f(m, m);
            const uint32_t scale = sb + kPad * 32 + j * (kPad * 36), sums = sb + kG_StageUnits * kPad * 36 + j * (kPad * 4);
#pragma unroll
            for (int g = 0; g < W / 4; ++g) {
                uint64_t x[2], s[2];
                lds_2x64(scale + 16u * g, x[0], x[1]);
                lds_2x64(sums + 16u * g, s[0], s[1]);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint64_t f = fma2(pack2((uint32_t)v[j][4 * g + 2 * i] + (1u << 19), (uint32_t)v[j][4 * g + 2 * i + 1] + (1u << 19)), sc2, c2);   // exact
                    const uint64_t t = fma2(m2, s[i], mul2(mul2(d2, x[i]), f));
                    sum[2 * g + i] = in_leaf ? add2(sum[2 * g + i], t) : t;
                }
            }
            if (++in_leaf == leaf) {
                in_leaf = 0;
                count_up<0>(n, sum, st, upper);
                ++n;
            }
        }
        tp.next();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cta(&sh.empty1[pos.r]);
        pos.next(false);
    }
    if (!ok) gemm_timeout(sh);
    return publish_sums<W>(status, sh, xch, q, part, lane, xphase, sum, ok);
}

// One output tile by one read-back warp: sums over its blocks, then into the exchange buffer.
template <class Policy, class Params, int COLG, int KG, int W>
__device__ __forceinline__ bool readback(const Params& p, const GemmWork& w, GemmShared& sh, uint32_t ring1, uint32_t ring2, float* xch, uint32_t tmem, int q,
                                         int part, int lane, RingPos& pos, TmemPos& tp, uint32_t& xphase) {
    pos.geometry(COLG * W <= 32);
    uint64_t acc2[W / 2];
#pragma unroll
    for (int i = 0; i < W / 2; ++i) acc2[i] = 0ull;
    const bool ok = readback_tile<COLG, KG, W, Policy::kAnyScale>(sh, ring1, ring2, tmem, p.status, uniform(w.nb), uniform(Policy::type(p, w)) < kTypeOperand, q, part, lane, pos, tp, acc2);
    return publish_sums<W, Policy::kAnyScale>(p.status, sh, xch, q, part, lane, xphase, acc2, ok);
}

template <class Policy, class Params, int COLG, int W>
__device__ __forceinline__ bool readback_as_gemv(const Params& p, const GemmWork& w, GemmShared& sh, uint32_t ring1, uint32_t ring2, float* xch, uint32_t tmem, int q,
                                                 int colg, int lane, RingPos& pos, TmemPos& tp, uint32_t& xphase) {
    pos.geometry(COLG * W <= 32);
    const int nb = uniform(w.nb), slice = uniform(Policy::slice(p, w));
    uint64_t total[W / 2];
    const bool ok = uniform(Policy::type(p, w)) == CHIMERE_TYPE_Q4_0
                        ? readback_ordered<CHIMERE_TYPE_Q4_0, COLG, W>(sh, ring1, ring2, tmem, p.status, nb, slice, q, colg, lane, pos, tp, total)
                        : readback_ordered<CHIMERE_TYPE_IQ3_S, COLG, W>(sh, ring1, ring2, tmem, p.status, nb, slice, q, colg, lane, pos, tp, total);
    return publish_sums<W>(p.status, sh, xch, q, colg, lane, xphase, total, ok);
}

// Slim tiles of packed weights: the read-back needs few of its warps and the two expander warps would be what bounds the kernel
// (1000 of 1490 cycles per stage with 16 columns), so parts 2 and 3 of the read-back warps expand instead, a row tile and
// two of a stage's four units each: warp x of eight.
template <class Policy, int MODE, class Params, int W>
__device__ __forceinline__ bool expand_slim(const Params& p, const GemmWork& w, GemmShared& sh, uint32_t ring1, uint32_t ring2, int x, int lane, RingPos& pos,
                                            TmemPos& tp, uint32_t& xphase) {
    const int type = uniform(Policy::type(p, w)), nb = uniform(w.nb);
    pos.geometry(1);
    if (tp.npad != W) { tp.npad = W; tp.slot = 0; tp.nslots = kG_TmemCols / (blocks_per_slot(W) * W); }
    const uint32_t t = x & 3, h = x >> 2;
    const uint32_t src = ring1 + t * kRawTile, dst = ring2 + h * (2 * kG_MmaTile) + t * 512 + lane * 16, rec = ring2 + 4096 + h * (2 * kG_MmaTile) + (t * 32 + lane) * 4;
    const int nstages = (nb + kG_StageUnits - 1) / kG_StageUnits;
    uint32_t d3 = 0u, sc3 = 0u;   // IQ3_S: this lane's row's scales of the super-block, kept over its two stages
    bool ok = true;
    for (int s = 0; s < nstages && ok; ++s) {
        const int u0 = stage_unit<MODE>(type, s);
        if (!mbar_wait(&sh.full1[pos.r], pos.par1()) || !mbar_wait(&sh.empty1[pos.lag()], pos.released(pos.lag()))) { ok = false; break; }
        const uint32_t raw = src + pos.slot1_off(), a = (uint32_t)pos.e * kG_ASlot;
        if (type == CHIMERE_TYPE_Q4_0) {
            const uint4 v0 = lds128(raw + (2 * h) * 576 + lane * 16), v1 = lds128(raw + (2 * h + 1) * 576 + lane * 16);
            const uint32_t e0 = lds16(raw + (2 * h) * 576 + 512 + lane * 2), e1 = lds16(raw + (2 * h + 1) * 576 + 512 + lane * 2);
            expand_unit<CHIMERE_TYPE_Q4_0>(v0, dst + a);
            expand_unit<CHIMERE_TYPE_Q4_0>(v1, dst + a + kG_MmaTile);
            sts_f32(rec + a, h2f(e0) * 0.0625f);
            sts_f32(rec + a + kG_MmaTile, h2f(e1) * 0.0625f);
        } else {
            const uint4 v0 = lds128(raw + (2 * h) * 512 + lane * 16), v1 = lds128(raw + (2 * h + 1) * 512 + lane * 16);
            if (!(s & 1)) {   // the scales came behind these units
                d3 = lds16(raw + 2048 + lane * 2);
                sc3 = lds32(raw + 2048 + 64 + lane * 4);
            }
            const uint32_t sc = sc3 >> (4 * (u0 & 4) + 8 * h);
            expand_unit<CHIMERE_TYPE_IQ3_S>(v0, dst + a);
            expand_unit<CHIMERE_TYPE_IQ3_S>(v1, dst + a + kG_MmaTile);
            sts_u32(rec + a, iq3s_word<MODE>(d3, sc & 15u));
            sts_u32(rec + a + kG_MmaTile, iq3s_word<MODE>(d3, (sc >> 4) & 15u));
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the MMAs read what ordinary stores wrote
        __syncwarp();
        if (lane == 0) mbar_arrive_cta(&sh.xfull2[pos.e]);
        // a stage is released by all of the read-back warps, and a tile's last one only when these have seen its accumulators complete: the
        // next tile may use the TMEM slots without them
        if (s + 1 == nstages && !mbar_wait(&sh.tfull[tp.slot], tp.par())) { ok = false; break; }
        if (lane == 0) mbar_arrive_cta(&sh.empty1[pos.r]);
        tp.next();
        pos.next(true);
    }
    if (ok && !mbar_wait(&sh.xempty, (xphase & 1u) ^ 1u)) ok = false;
    ++xphase;
    if (!ok) gemm_timeout(sh);
    if (lane == 0) mbar_arrive_cta(&sh.xfull);   // nothing of this warp's to store
    return ok;
}

// Warps 4..7: what happens to a tile's sums, while the read-back warps are at the next tile.
template <class Policy, int MODE, class Params>
__device__ __forceinline__ bool store_tile(const Params& p, const GemmWork& w, GemmShared& sh, const float* xch, int ew, int lane, uint32_t& xphase) {
    const bool ok = mbar_wait(&sh.xfull, xphase & 1u);
    ++xphase;
    if (!ok) { gemm_timeout(sh); return false; }
    if (MODE != kPlain || w.npad == 128) Policy::template store<1, MODE>(p, w, xch, ew, lane);
    else if (w.npad == 64 || Policy::type(p, w) < kTypeOperand) Policy::template store<2, kPlain>(p, w, xch, ew, lane);
    else Policy::template store<4, kPlain>(p, w, xch, ew, lane);
    __syncwarp();
    if (lane == 0) mbar_arrive_cta(&sh.xempty);
    return true;
}

// The next tile of the schedule ring, for every warp but the scheduler's own; negative: no more (or a wait ran out).
__device__ __forceinline__ int take_tile(GemmShared& sh, int32_t* status, uint32_t& tn, int lane) {
    const int slot = (int)(tn % kG_Sched);
    if (!mbar_wait(&sh.sfull[slot], (tn / kG_Sched) & 1u)) { gemm_timeout(sh); return -1; }
    const int idx = *reinterpret_cast<volatile int*>(&sh.sched[slot]);
    __syncwarp();
    if (lane == 0) mbar_arrive_cta(&sh.sempty[slot]);
    ++tn;
    return idx;
}

template <class Policy, class Params, int MODE = kPlain>
__global__ void __launch_bounds__(kG_Threads, 1) gemm_i8_kernel(const Params p, int32_t* tile_counter) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ GemmShared sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = uniform(tid >> 5);
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* ring1 = smem + kG_ConstBytes;
    uint8_t* ring2 = ring1 + kG_RingBytes;
    float* xch = reinterpret_cast<float*>(ring2 + kG_ASlots * kG_ASlot);

    if (tid == 0) {
        for (int i = 0; i < kG_RingSlotsSlim; ++i) { mbar_init(&sh.full1[i], 1); mbar_init(&sh.empty1[i], kG_RbWarps); }
        for (int i = 0; i < kG_ASlots; ++i) { mbar_init(&sh.xfull2[i], kG_SlimExpWarps); }
        for (int i = 0; i < kG_TmemSlots; ++i) { mbar_init(&sh.tfull[i], 1); mbar_init(&sh.tempty[i], kG_RbWarps); }
        for (int i = 0; i < kG_Sched; ++i) { mbar_init(&sh.sfull[i], 1); mbar_init(&sh.sempty[i], 1 + kG_ExpWarps + kG_EpiWarps + kG_RbWarps); }
        mbar_init(&sh.xfull, kG_RbWarps); mbar_init(&sh.xempty, kG_EpiWarps);
        sh.failed = 0;
        mbar_fence_init();
    }
    for (int i = tid; i < kG_ConstBytes / 4; i += kG_Threads) reinterpret_cast<uint32_t*>(smem)[i] = 0x80808080u;   // int8 -128
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_base)), "r"(kG_TmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_base;
    // The set-up above may run while the kernel that fills the operands finishes.  The tiles with minimums are launched behind the others'
    // kernel, whose CTAs have all waited for that already; their CTAs come in as those run out of tiles, and wait for that kernel's end
    // before they go (below), so that whoever waits for this grid has both.
    if (MODE != kMin) griddep_wait();
    if (tid == 0) griddep_launch();

    // The read-back warps and the others take separate paths from here on, each with its own share of the registers.
    if (warp >= kG_FirstRb) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kG_RegsRb));
        const int q = warp & 3, part = (warp - kG_FirstRb) >> 2;   // TMEM lane quarter this warp may read; its share of columns and stages
        RingPos pos;
        TmemPos tp;
        uint32_t tn = 0, xphase = 0;
        int idx;
        bool ok = true;
        while (ok && (idx = take_tile(sh, p.status, tn, lane)) >= 0) {
            GemmWork w;
            Policy::template work<MODE>(p, idx, w);
            const uint32_t r1 = smem_u32(ring1), r2 = smem_u32(ring2);
            if (MODE == kOrdered) {
                switch (uniform(w.npad)) {
                    case 64: ok = readback_as_gemv<Policy, Params, 4, 16>(p, w, sh, r1, r2, xch, tmem, q, part, lane, pos, tp, xphase); break;
                    case 32:
                        if (part < 2) ok = readback_as_gemv<Policy, Params, 2, 16>(p, w, sh, r1, r2, xch, tmem, q, part, lane, pos, tp, xphase);
                        else ok = expand_slim<Policy, MODE, Params, 32>(p, w, sh, r1, r2, warp - kG_FirstRb - 8, lane, pos, tp, xphase);
                        break;
                    default:
                        if (part < 2) ok = readback_as_gemv<Policy, Params, 2, 8>(p, w, sh, r1, r2, xch, tmem, q, part, lane, pos, tp, xphase);
                        else ok = expand_slim<Policy, MODE, Params, 16>(p, w, sh, r1, r2, warp - kG_FirstRb - 8, lane, pos, tp, xphase);
                        break;
                }
                continue;
            }
            if (MODE == kMin) {
                const int nb = uniform(w.nb);
                ok = readback_min(sh, r1, r2, xch, tmem, p.status, nb, Policy::tree_order(p) ? nb >> 5 : nb, q, part, lane, pos, tp, xphase);
                continue;
            }
            switch (uniform(w.npad)) {
                case 128: ok = readback<Policy, Params, 4, 1, 32>(p, w, sh, r1, r2, xch, tmem, q, part, lane, pos, tp, xphase); break;
                case 64: ok = readback<Policy, Params, 2, 2, 32>(p, w, sh, r1, r2, xch, tmem, q, part, lane, pos, tp, xphase); break;
                case 32:
                    if (uniform(Policy::type(p, w)) >= kTypeOperand) ok = readback<Policy, Params, 1, 4, 32>(p, w, sh, r1, r2, xch, tmem, q, part, lane, pos, tp, xphase);
                    else if (part < 2) ok = readback<Policy, Params, 1, 2, 32>(p, w, sh, r1, r2, xch, tmem, q, part, lane, pos, tp, xphase);
                    else ok = expand_slim<Policy, MODE, Params, 32>(p, w, sh, r1, r2, warp - kG_FirstRb - 8, lane, pos, tp, xphase);
                    break;
                default:
                    if (uniform(Policy::type(p, w)) >= kTypeOperand) ok = readback<Policy, Params, 1, 4, 16>(p, w, sh, r1, r2, xch, tmem, q, part, lane, pos, tp, xphase);
                    else if (part < 2) ok = readback<Policy, Params, 1, 2, 16>(p, w, sh, r1, r2, xch, tmem, q, part, lane, pos, tp, xphase);
                    else ok = expand_slim<Policy, MODE, Params, 16>(p, w, sh, r1, r2, warp - kG_FirstRb - 8, lane, pos, tp, xphase);
                    break;
            }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kG_RegsAux));
        RingPos pos;
        uint32_t tn = 0;
        bool ok = true;
        if (warp == 0) {
            // ------------------------------ tile scheduler + operand producer ------------------------------
            bool skipped = false;   // warps 2..3 sat out the tile before
            while (ok) {
                GemmWork w;
                int idx = 0, ws;
                do {   // a skipped index costs one more atomic
                    if (lane == 0) idx = atomicAdd(tile_counter, 1);
                    idx = __shfl_sync(0xffffffffu, idx, 0);
                    ws = Policy::template work<MODE>(p, idx, w);
                } while (ws == kWorkSkip);
                if (ws == kWorkOk) {
                    // Parity tells a barrier's phases apart only for those who are at most one behind, and warps 2..3 saw nothing of the tiles
                    // that they sat out: they learn of a tile of theirs when every stage before it has been read back.
                    const bool expand = warps23_expand<MODE>(uniform(Policy::type(p, w)), uniform(w.npad) <= 32);
                    if (expand && skipped)
                        for (int r = 0; r < pos.slots1() && ok; ++r)
                            if (!mbar_wait(&sh.empty1[r], pos.released(r))) { gemm_timeout(sh); ok = false; }
                    if (!ok) break;
                    skipped = !expand;
                }
                const int slot = (int)(tn % kG_Sched);
                if (!mbar_wait(&sh.sempty[slot], ((tn / kG_Sched) & 1u) ^ 1u)) { gemm_timeout(sh); ok = false; break; }
                if (lane == 0) {
                    sh.sched[slot] = ws == kWorkEnd ? -1 : idx;
                    mbar_arrive_cta(&sh.sfull[slot]);   // (release: the index is visible to whoever sees the arrival)
                }
                ++tn;
                if (ws == kWorkEnd) break;
                ok = produce_tile<Policy, MODE>(p, w, sh, ring1, ring2, pos, lane);
            }
            if (!ok)   // a wait ran out: the copies already asked for have to land before this CTA's memory goes away
                for (int r = 0; r < pos.slots1(); ++r) mbar_wait(&sh.full1[r], pos.released(r));
        } else {
            TmemPos tp;
            uint32_t xphase = 0;
            int idx;
            while (ok && (idx = take_tile(sh, p.status, tn, lane)) >= 0) {
                GemmWork w;
                Policy::template work<MODE>(p, idx, w);
                const uint32_t r1 = smem_u32(ring1), r2 = smem_u32(ring2);
                if (warp == 1) {
                    const uint32_t cst = smem_u32(smem);
                    if (MODE == kMin) ok = mma_tile<Policy, MODE, 32>(p, w, sh, cst, r1, r2, tmem, pos, tp, lane);
                    else switch (uniform(w.npad)) {
                        case 128: if (MODE == kPlain) ok = mma_tile<Policy, MODE, 128>(p, w, sh, cst, r1, r2, tmem, pos, tp, lane); break;
                        case 64: ok = mma_tile<Policy, MODE, 64>(p, w, sh, cst, r1, r2, tmem, pos, tp, lane); break;
                        case 32: ok = mma_tile<Policy, MODE, 32>(p, w, sh, cst, r1, r2, tmem, pos, tp, lane); break;
                        default: ok = mma_tile<Policy, MODE, 16>(p, w, sh, cst, r1, r2, tmem, pos, tp, lane); break;
                    }
                } else if (warp < kG_FirstEpi) {
                    ok = expand_tile<Policy, MODE>(p, w, sh, r1, r2, pos, warp - 2, lane);
                } else {
                    ok = store_tile<Policy, MODE>(p, w, sh, xch, warp - kG_FirstEpi, lane, xphase);
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kG_TmemCols) : "memory");
    }
    if (tid == 0 && sh.failed && p.status) atomicOr(p.status, kStatusWaitTimeout);
    if (MODE == kMin) griddep_wait();
}

// ------------------------------------------------------------------ policies ----
// plain fp32 tile store: out[(row0 + r) * ldo + col0 + c] = D[r][c]  (the primitive; operands in the mma128 form)
struct PlainPolicy {
    static constexpr bool kAnyScale = true;
    template <int>
    __device__ static __forceinline__ int work(const GemmParams& p, int idx, GemmWork& w) {
        if (idx >= p.n_items) return kWorkEnd;
        const GemmItem it = p.items[idx];
        w.b = p.b_base + it.b_offset;
        w.nb = p.nblocks; w.n_valid = it.n_valid; w.npad = 128;
        w.expert = idx; w.shared = 0; w.rt = it.rows_valid; w.start = 0; w.col16 = 0;
        w.aux0 = it.out_row0; w.aux1 = it.out_col0;
        return kWorkOk;
    }
    __device__ static __forceinline__ int type(const GemmParams&, const GemmWork&) { return kTypeOperand; }
    __device__ static __forceinline__ int slice(const GemmParams&, const GemmWork&) { return 1; }
    __device__ static __forceinline__ bool tree_order(const GemmParams&) { return false; }
    __device__ static __forceinline__ RowTiles rows(const GemmParams& p, const GemmWork& w) { return RowTiles{p.a_base + p.items[w.expert].a_offset, nullptr, 0, 0, 0}; }
    template <int KG, int MODE>
    __device__ static __forceinline__ void store(const GemmParams& p, const GemmWork& w, const float* xch, int ew, int lane) {
        for (int r = ew; r < w.rt; r += kG_EpiWarps)   // (all tiles of the primitive are 128 columns wide: one share)
            for (int c = lane; c < w.n_valid; c += 32) p.out[(size_t)(w.aux0 + r) * p.ldo + w.aux1 + c] = xch[c * 128 + r];
    }
};

// Token tiles (built on the device after routing): {expert (-1 = shared expert), start, pairs, first column / 16}; word 0 of
// the list = number of tiles, words 4 and 5 = the tile counters of the two GEMM launches (zero when the list is built).
// Routed tile: pairs perm[start .. start + n); shared tile: tokens start .. .  A tile of n pairs is tile_width(n) columns wide.
constexpr int kTileHeader = 8;
__device__ __forceinline__ int tile_width(int n) { return n <= 16 ? 16 : n <= 32 ? 32 : n <= 64 ? 64 : 128; }

// What the gate/up and the down launch share: the tile list and where a row tile's weights are.
struct MoePolicy {
    static constexpr bool kAnyScale = false;   // (ggml's scales are f16)
    template <int MODE>
    __device__ static __forceinline__ int work(const PrefillGemmParams& p, int idx, GemmWork& w) {
        if (MODE == kMin) {   // shared-expert tiles of 32 tokens; word 1 of the list: their first column / 16
            const PrefillGemmMats& m = p.m[1];
            const int j = idx / m.row_tiles, t0 = j * 32;
            if (t0 >= p.T) return kWorkEnd;
            w.shared = 1; w.expert = 0; w.rt = idx - j * m.row_tiles;
            w.nb = m.ncols >> 5; w.n_valid = min(32, p.T - t0); w.npad = 32;
            w.start = t0; w.col16 = __ldcg(p.tiles + 1) + 2 * j;
            w.b = p.b_tiles + (size_t)w.col16 * p.b_col16_bytes;
            w.aux0 = w.aux1 = 0;
            return kWorkOk;
        }
        const int j = idx / p.row_tiles_max, rt = idx - j * p.row_tiles_max;
        if (j >= __ldcg(p.tiles)) return kWorkEnd;
        const int4 t = __ldcg(reinterpret_cast<const int4*>(p.tiles + kTileHeader) + j);
        w.shared = t.x < 0 ? 1 : 0;
        const PrefillGemmMats& m = p.m[w.shared];
        if (rt >= m.row_tiles) return kWorkSkip;
        w.expert = t.x < 0 ? 0 : t.x;
        w.nb = m.ncols >> 5; w.n_valid = t.z; w.npad = tile_width(t.z);
        w.rt = rt; w.start = t.y; w.col16 = t.w;
        w.b = p.b_tiles + (size_t)t.w * p.b_col16_bytes;
        w.aux0 = w.aux1 = 0;
        return kWorkOk;
    }
    __device__ static __forceinline__ int type(const PrefillGemmParams& p, const GemmWork& w) { return p.m[w.shared].type; }
    __device__ static __forceinline__ int slice(const PrefillGemmParams& p, const GemmWork& w) { return p.m[w.shared].slice; }
    __device__ static __forceinline__ bool tree_order(const PrefillGemmParams& p) { return p.shared_sums != 0; }   // (set for the gate/up launch)
    // gated: two 32-row tiles of the gate matrix and the same two of the up matrix; else four of the one matrix
    __device__ static __forceinline__ RowTiles rows(const PrefillGemmParams& p, const GemmWork& w) {
        const PrefillGemmMats& m = p.m[w.shared];
        RowTiles r{m.w0 + (size_t)w.expert * m.stride0, nullptr, (int)m.tile_bytes, 0, 0};
        if (m.type >= kTypeOperand) { r.src0 += (size_t)w.rt * w.nb * (m.type == kTypeOperand ? kG_MmaTile : kOperandMinStage / kG_StageUnits); return r; }
        if (p.dual) {
            r.src0 += (size_t)(2 * w.rt) * m.tile_bytes;
            r.src1 = m.w1 + (size_t)w.expert * m.stride1 + (size_t)(2 * w.rt) * m.tile_bytes;
            r.n0 = r.n1 = min(2, m.rows32 - 2 * w.rt);
        } else {
            r.src0 += (size_t)(4 * w.rt) * m.tile_bytes;
            r.src1 = r.src0 + 2 * m.tile_bytes;
            r.n0 = min(2, m.rows32 - 4 * w.rt);
            r.n1 = max(0, min(2, m.rows32 - 4 * w.rt - 2));
        }
        return r;
    }
};

// sums of the K shares, shares in order
template <int KG>
__device__ __forceinline__ float xch_sum(const float* xch, int npad, int row, int c) {
    float v = xch[c * 128 + row];
#pragma unroll
    for (int k = 1; k < KG; ++k) v += xch[(k * npad + c) * 128 + row];
    return v;
}

// gate/up: A tile = 64 gate rows | 64 up rows of the same 64 intermediate rows (or 128 up rows when there is no gate).  The
// activation is quantised to Q8_1 (32 consecutive rows = one warp) straight into the down GEMM's token tile.  A warp takes
// a 32-row block of the intermediate and every second or every column of the tile, two columns at a time so that the
// divisions of one hide the other's.
struct GateUpPolicy : MoePolicy {
    template <int KG, int MODE>
    __device__ static __forceinline__ void store(const PrefillGemmParams& p, const GemmWork& w, const float* xch, int ew, int lane) {
        const int nrb = p.dual ? 2 : 4, rb = ew & (nrb - 1), blk = w.rt * nrb + rb;
        if (blk >= p.m[w.shared].rows32) return;     // (the last row tile may be partly filled)
        const int cstep = kG_EpiWarps / nrb, r = rb * 32 + lane;
        const bool sums = MODE == kMin;   // the down matrix has minimums too: it wants the blocks' sums
        uint8_t* tile = p.out_tiles + (size_t)w.col16 * p.out_col16_bytes;
        uint8_t* dst = sums ? tile + (size_t)(blk >> 2) * (w.npad * 160) + (blk & 3) * (w.npad * 36) : tile + (size_t)blk * (w.npad * 36);
        float* sdst = reinterpret_cast<float*>(tile + (size_t)(blk >> 2) * (w.npad * 160) + w.npad * 144 + (blk & 3) * (w.npad * 4));
        int8_t* qdst = reinterpret_cast<int8_t*>(dst) + (lane >> 4) * (w.npad * 16) + (lane & 15);
        float* ddst = reinterpret_cast<float*>(dst + w.npad * 32);
        for (int c = ew / nrb; c < w.n_valid; c += 2 * cstep) {
            float v[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int ci = min(c + i * cstep, w.n_valid - 1);
                const float a = xch_sum<KG>(xch, w.npad, r, ci);
                if (p.dual) { const float u = xch_sum<KG>(xch, w.npad, r + 64, ci); v[i] = MODE != kPlain ? silu_mul_ref(a, u) : silu_mul_fast(a, u); }
                else { const float t = fmaxf(a, 0.0f); v[i] = t * t; }
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int ci = c + i * cstep;
                float d;
                const int8_t qv = q8_1_warp(v[i], d);
                if (ci < w.n_valid) {
                    qdst[(ci >> 3) * 128 + (ci & 7) * 16] = qv;
                    if (lane == 0) ddst[ci] = __half2float(__float2half(d));
                }
                if (sums || p.inter_q8) {
                    float sum = v[i];
#pragma unroll
                    for (int k = 16; k > 0; k >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, k);
                    const __half sh = __float2half(sum);
                    if (sums && lane == 0 && ci < w.n_valid) sdst[ci] = __half2float(sh);
                    if (p.inter_q8 && ci < w.n_valid) {   // the decode entry's rows of intermediates
                        const int row = w.shared ? p.T * p.top_k + w.start + ci : __ldcg(p.perm + w.start + ci);
                        uint8_t* tap = p.inter_q8 + (size_t)row * p.inter_stride + (size_t)blk * kQ81Bytes;
                        reinterpret_cast<int8_t*>(tap)[4 + lane] = qv;
                        p.inter_q[(size_t)row * p.inter_q_stride + blk * 32 + lane] = qv;
                        if (lane == 0) {
                            *reinterpret_cast<__half2*>(tap) = __halves2half2(__float2half(d), sh);
                            p.inter_d[(size_t)row * p.inter_d_stride + blk] = __half2float(__float2half(d));
                        }
                    }
                }
            }
        }
        // Token columns past n_valid of the tile are left as they are: the down GEMM never stores them, and every
        // column's sums depend on that column alone.
    }
};

// down: rows of H; the tile's columns are pairs, written to pair_out[pair row][H].  A warp stores the 128 rows of every fourth
// column, four rows per lane (H is a multiple of 32).  The shared expert's rows have a place of their own.
struct DownPolicy : MoePolicy {
    template <int KG, int MODE>
    __device__ static __forceinline__ void store(const PrefillGemmParams& p, const GemmWork& w, const float* xch, int ew, int lane) {
        const bool rows = w.rt * 128 + lane * 4 < p.H;
        float* out = (w.shared ? p.shared_out : p.pair_out) + w.rt * 128 + lane * 4;
        const float* x = xch + lane * 4;
        for (int c0 = 0; c0 < w.n_valid; c0 += 128) {
            // this lane's pair rows: of columns ew + 4 * lane
            const int cl = c0 + ew + 4 * lane;
            int prow = 0;
            if (cl < w.n_valid) prow = w.shared ? w.start + cl : __ldcg(p.perm + w.start + cl);
            const int n = min(32, (w.n_valid - c0 - ew + 3) >> 2);
#pragma unroll 4
            for (int i = 0; i < n; ++i) {
                const int c = c0 + ew + 4 * i;
                float4 v = *reinterpret_cast<const float4*>(x + c * 128);
#pragma unroll
                for (int k = 1; k < KG; ++k) {
                    const float4 u = *reinterpret_cast<const float4*>(x + (k * w.npad + c) * 128);
                    v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
                }
                const int row = __shfl_sync(0xffffffffu, prow, i);
                if (rows) *reinterpret_cast<float4*>(out + (size_t)row * p.H) = v;
            }
        }
    }
};

// [rows][cols] int8 + [rows][cols/32] f32 scales -> mma128 tiles (rows padded with zeros to a multiple of 128).
// One thread per (row, block).
__global__ void pack_mma128_kernel(const int8_t* q, const float* scales, uint8_t* out, int rows, int cols) {
    const int nb = cols >> 5;
    const int rows_pad = (rows + 127) & ~127;
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)rows_pad * nb) return;
    const int row = (int)(idx % rows_pad), b = (int)(idx / rows_pad);
    const int tile = row >> 7, r = row & 127;
    uint8_t* dst = out + ((size_t)tile * nb + b) * kG_MmaTile;
    uint4 lo = make_uint4(0, 0, 0, 0), hi = lo;
    float sc = 0.0f;
    if (row < rows) {
        const uint4* src = reinterpret_cast<const uint4*>(q + (size_t)row * cols + b * 32);
        lo = src[0]; hi = src[1];
        sc = scales[(size_t)row * nb + b];
    }
    *reinterpret_cast<uint4*>(dst + (r >> 3) * 128 + (r & 7) * 16) = lo;          // k 0..15
    *reinterpret_cast<uint4*>(dst + 2048 + (r >> 3) * 128 + (r & 7) * 16) = hi;   // k 16..31
    *reinterpret_cast<float*>(dst + 4096 + r * 4) = sc;
}

cudaError_t launch_pack_mma128(const int8_t* q, const float* scales, uint8_t* out, int rows, int cols, cudaStream_t stream) {
    const int64_t n = (int64_t)((rows + 127) & ~127) * (cols / 32);
    if (n <= 0) return cudaSuccess;
    pack_mma128_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(q, scales, out, rows, cols);
    return cudaGetLastError();
}

// persistent CTAs: one per SM of the current device, or fewer when there are fewer tiles
static int gemm_grid(int n_items) {
    const int n_sm = sm_count();
    return n_items < n_sm ? n_items : n_sm;
}
template <class Policy, int MODE = kPlain, class Params>
static cudaError_t launch_gemm(const Params& p, int n_items, int32_t* counter, cudaStream_t stream) {
    static bool attr_done[64] = {};
    cudaError_t e = max_smem_once(gemm_i8_kernel<Policy, Params, MODE>, (int)kG_Smem, attr_done);
    if (e != cudaSuccess) return e;
    return launch_pdl(gemm_i8_kernel<Policy, Params, MODE>, dim3(gemm_grid(n_items)), kG_Threads, kG_Smem, stream, p, counter);
}

// tile_counter: one int32 of device memory that is zero when the kernel starts (it ends at n_items + the number of CTAs)
cudaError_t launch_gemm_i8_f32(const GemmParams& p_in, int n_items, int32_t* tile_counter, cudaStream_t stream) {
    if (n_items <= 0) return cudaSuccess;
    GemmParams p = p_in;
    p.n_items = n_items;
    return launch_gemm<PlainPolicy>(p, n_items, tile_counter, stream);
}

// The tile list's header words 4 (gate/up) and 5 (down) are the launches' tile counters; build_tiles_kernel zeroes them.
cudaError_t launch_prefill_gemm(const PrefillGemmParams& p, bool down, int n_tiles_max, bool min_only, cudaStream_t stream) {
    const int n_items = n_tiles_max * p.row_tiles_max;
    if (n_items <= 0) return cudaSuccess;
    int32_t* counter = const_cast<int32_t*>(p.tiles) + (down ? 5 : 4);
    cudaError_t e = cudaSuccess;
    if (min_only) {}
    else if (p.as_gemv) e = down ? launch_gemm<DownPolicy, kOrdered>(p, n_items, counter, stream) : launch_gemm<GateUpPolicy, kOrdered>(p, n_items, counter, stream);
    else e = down ? launch_gemm<DownPolicy>(p, n_items, counter, stream) : launch_gemm<GateUpPolicy>(p, n_items, counter, stream);
    if (e == cudaSuccess && p.m[1].type == kTypeOperandMin) {   // (words 6 / 7: these launches' counters)
        const int n_min = (p.T + 31) / 32 * p.m[1].row_tiles;
        e = down ? launch_gemm<DownPolicy, kMin>(p, n_min, counter + 2, stream) : launch_gemm<GateUpPolicy, kMin>(p, n_min, counter + 2, stream);
    }
    return e;
}

// ------------------------------------------------------------------ tensor-pipe probe ----
// What the int8 tensor pipe can do when nothing is read back: every CTA (one per SM) keeps issuing
// tcgen05.mma kind::i8 (M 128, N 128 or 256, K 32) on operands resident in shared memory, accumulating in TMEM,
// with a commit every 64 instructions and a bounded wait on the last one.  Timed from the host with events, this
// is the denominator the prefill numbers are stated against (2 * 128 * N * 32 operations per instruction).
__global__ void __launch_bounds__(128, 1) mma_i8_probe_kernel(int n_mma, int n_cols, int n_acc, int32_t* status) {
    extern __shared__ __align__(1024) uint8_t smem[];   // A: 128 x 32 int8 (4096 B), B: n_cols x 32 int8
    __shared__ __align__(8) uint64_t s_bar[2];   // commit groups alternate between the two
    __shared__ uint32_t s_tmem;
    const int tid = threadIdx.x, warp = tid >> 5;
    for (int i = tid; i < (4096 + n_cols * 32) / 4; i += blockDim.x)
        reinterpret_cast<uint32_t*>(smem)[i] = 0x9E3779B9u * (uint32_t)(i + 1 + blockIdx.x * 977);   // any bytes will do
    if (tid == 0) { mbar_init(&s_bar[0], 1); mbar_init(&s_bar[1], 1); mbar_fence_init(); }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the operands were written by ordinary stores
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    if (tid == 0) {
        const uint32_t sa = smem_u32(smem), sb = sa + 4096;
        const uint32_t lbo_b = (uint32_t)n_cols * 16u;   // K halves of B are n_cols / 8 row groups of 128 bytes apart
        const uint64_t adesc = smem_desc_kmajor(sa, 2048);
        const uint64_t bdesc = (uint64_t)((sb & 0x3FFFFu) >> 4) | ((uint64_t)(lbo_b >> 4) << 16) | ((uint64_t)(128u >> 4) << 32) | (1ull << 46);
        const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | (((uint32_t)n_cols >> 3) << 17) | ((128u >> 4) << 24);
        auto mma = [&](uint32_t d, uint32_t acc) {
            asm volatile(
                "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
                ::"r"(d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u) : "memory");
        };
        // accumulators taken in turn (n_acc of them, n_cols columns each); groups of 64 instructions per commit
        uint32_t dcol[4];
        for (int j = 0; j < 4; ++j) dcol[j] = tmem + (uint32_t)((j % n_acc) * n_cols);
        const int groups = (n_mma + 63) / 64;
        bool ok = true;
        for (int g = 0; g < groups && ok; ++g) {
#pragma unroll 4
            for (int j = 0; j < 64; j += 4) {
                mma(dcol[0], g > 0 || j >= 4 ? 1u : 0u);
                mma(dcol[1], g > 0 || j >= 4 ? 1u : 0u);
                mma(dcol[2], g > 0 || j >= 4 ? 1u : 0u);
                mma(dcol[3], g > 0 || j >= 4 ? 1u : 0u);
            }
            tc_commit(&s_bar[g & 1]);
            // at most two commit groups in flight: wait for the one before the one just issued
            if (g >= 1 && !mbar_wait(&s_bar[(g - 1) & 1], ((g - 1) >> 1) & 1)) { if (status) atomicOr(status, kStatusWaitTimeout); ok = false; }
        }
        if (ok && groups >= 1 && !mbar_wait(&s_bar[(groups - 1) & 1], ((groups - 1) >> 1) & 1) && status) atomicOr(status, kStatusWaitTimeout);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// Returns the number of CTAs launched (each issues n_mma instructions, rounded up to a multiple of 64), or a negative CUDA error.
int launch_mma_i8_probe(int n_mma, int n_cols, int n_acc, int32_t* status, cudaStream_t stream) {
    const int ctas = gemm_grid(1 << 30);
    const size_t smem = 4096 + (size_t)n_cols * 32 + 1024;
    mma_i8_probe_kernel<<<ctas, 128, smem, stream>>>(n_mma, n_cols, n_acc, status);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? ctas : -100 - (int)e;
}

// ------------------------------------------------------------------ prefill plumbing kernels ----
// ggml Q8_0 blocks -> mma128 tiles: int8 values in the MMA's operand order and f32 block scales.
// dst row of source row r: plain (mode 0), gate half (mode 1: (r/64)*128 + r%64) or up half (mode 2: ... + 64).
// One thread per (row, block); blockIdx.y = expert.
__global__ void pack_mma128_q8_0_kernel(const uint8_t* raw, uint8_t* out, int nrows, int ncols, int mode, int64_t raw_stride, int64_t out_stride) {
    const int nb = ncols >> 5;
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)nrows * nb) return;
    const int r = (int)(idx % nrows), b = (int)(idx / nrows);
    int w[8], mul;
    float dw;
    using U = Unit<CHIMERE_TYPE_Q8_0>;
    U::load(raw + (size_t)blockIdx.y * raw_stride + (size_t)r * U::row_bytes(ncols), b, nullptr, w, dw, mul);
    const int dr = mode == 0 ? r : (r >> 6) * 128 + (r & 63) + (mode == 2 ? 64 : 0);
    const int tile = dr >> 7, rr = dr & 127;
    uint8_t* dst = out + (size_t)blockIdx.y * out_stride + ((size_t)tile * nb + b) * kG_MmaTile;
    *reinterpret_cast<uint4*>(dst + (rr >> 3) * 128 + (rr & 7) * 16) = make_uint4(w[0], w[1], w[2], w[3]);
    *reinterpret_cast<uint4*>(dst + 2048 + (rr >> 3) * 128 + (rr & 7) * 16) = make_uint4(w[4], w[5], w[6], w[7]);
    *reinterpret_cast<float*>(dst + 4096 + rr * 4) = dw;
}

cudaError_t launch_pack_mma128_q8_0(const void* raw, void* out, int n_mats, int nrows, int ncols, int mode, int64_t raw_stride, int64_t out_stride,
                                    cudaStream_t stream) {
    if (n_mats <= 0) return cudaSuccess;
    const int64_t n = (int64_t)nrows * (ncols / 32);
    pack_mma128_q8_0_kernel<<<dim3((unsigned)((n + 255) / 256), (unsigned)n_mats), 256, 0, stream>>>((const uint8_t*)raw, (uint8_t*)out, nrows, ncols, mode,
                                                                                                     raw_stride, out_stride);
    return cudaGetLastError();
}

// After routing: the token tiles of every expert with at least gemm_min pairs (and of the shared expert), and, if `list` is given, the
// GEMV work list of the others (gemm_min <= kMaxGroupTokens + 1).  One CTA of 256 threads,
// thread e = expert e.  Wide tiles come first and the narrow ones last, so that the persistent GEMM CTAs, which take tiles
// in order, end on cheap ones; within a width the shared expert's tile leads.  Tiles per width are counted with one scan
// (a 64-bit word of counters, 28 bits for the full tiles' width and 12 for each narrower one, of which an expert has at most one tile), and a tile's first column follows from its place, because all tiles of a width
// are equally wide.
__device__ __forceinline__ int width_class(int n) { return n > 64 ? 0 : n > 32 ? 1 : n > 16 ? 2 : 3; }
__device__ __forceinline__ int width_shift(int k) { return k <= 0 ? 0 : 16 + 12 * k; }    // k: classes below the full tiles'
__device__ __forceinline__ int width_count(uint64_t counts, int k) { return (int)(counts >> width_shift(k)) & (k <= 0 ? (1 << 28) - 1 : 0xFFF); }
__global__ void __launch_bounds__(256) build_tiles_kernel(const int32_t* offsets, const int32_t* perm, int32_t* tiles, int32_t* list, int E, int T,
                                                          int has_shared, int gemm_min, int shared_32, int widest) {
    __shared__ uint64_t scan[8];
    __shared__ int scan_n[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    griddep_wait();
    if (tid == 0) griddep_launch();
    const int pairs = tid < E ? offsets[tid + 1] - offsets[tid] : 0, off = tid < E ? offsets[tid] : 0;
    // experts of fewer than gemm_min pairs go to the GEMV kernels, one work entry each
    const bool small = pairs > 0 && pairs < gemm_min;
    const int cnt = small ? 0 : pairs;
    if (list) {
        const unsigned m = __ballot_sync(0xffffffffu, small);
        if (lane == 0) scan_n[warp] = __popc(m);
        __syncthreads();
        int first = __popc(m & ((1u << lane) - 1u)), total = 0;
        for (int w = 0; w < 8; ++w) { if (w < warp) first += scan_n[w]; total += scan_n[w]; }
        if (small) {
            int* ent = list + kListHeader + kListEntry * first;
            ent[0] = tid; ent[1] = off; ent[2] = pairs; ent[3] = 0;
            for (int j = 0; j < kMaxGroupTokens; ++j) ent[4 + j] = j < pairs ? perm[off + j] : 0;
        }
        if (tid == 0) { list[0] = total; list[1] = total; list[2] = 0; list[3] = 0; }
    }
    const int full = widest, fshift = widest == 128 ? 7 : 6, kf = 7 - fshift;   // columns of a full tile, their width's place in the list
    const int nf = cnt >> fshift, rem = cnt & (full - 1);
    auto one = [&](int n) { return 1ull << width_shift(width_class(n) - kf); };
    const uint64_t own = (uint64_t)nf + (rem ? one(rem) : 0ull);
    uint64_t incl = own;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const uint64_t a = __shfl_up_sync(0xffffffffu, incl, s);
        if (lane >= s) incl += a;
    }
    if (lane == 31) scan[warp] = incl;
    __syncthreads();
    uint64_t before = incl - own, total = 0;
    for (int w = 0; w < 8; ++w) { if (w < warp) before += scan[w]; total += scan[w]; }
    // the shared expert's tiles: 128 columns and a rest, or (shared_32) tiles of 32 that are not on the list, their columns behind all
    // others'
    const int sh_full = has_shared && !shared_32 ? T >> fshift : 0, sh_rem = has_shared && !shared_32 ? T & (full - 1) : 0;
    const uint64_t shared = (uint64_t)sh_full + (sh_rem ? one(sh_rem) : 0ull);
    total += shared;
    before += shared;   // the shared expert's tiles lead every width
    int first[5], col16[5];   // first tile and first column / 16 of each width
    first[0] = 0; col16[0] = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int n = k < kf ? 0 : width_count(total, k - kf);
        first[k + 1] = first[k] + n;
        col16[k + 1] = col16[k] + n * (8 >> k);
    }
    int4* tv = reinterpret_cast<int4*>(tiles + kTileHeader);
    auto put = [&](int k, int i, int expert, int start, int n) { tv[first[k] + i] = make_int4(expert, start, n, col16[k] + i * (8 >> k)); };
    for (int i = tid; i < sh_full; i += 256) put(kf, i, -1, i * full, full);
    if (tid == 0 && sh_rem) put(width_class(sh_rem), width_class(sh_rem) == kf ? sh_full : 0, -1, sh_full * full, sh_rem);
    const int f0 = width_count(before, 0);
    for (int i = 0; i < nf; ++i) put(kf, f0 + i, tid, off + i * full, full);
    if (rem) {
        const int k = width_class(rem);
        put(k, width_count(before, k - kf) + (k == kf ? nf : 0), tid, off + nf * full, rem);
    }
    if (tid == 0) {
        tiles[0] = first[4]; tiles[1] = col16[4]; tiles[2] = 0; tiles[3] = 0;
        tiles[4] = 0; tiles[5] = 0; tiles[6] = 0; tiles[7] = 0;   // the two GEMM launches' tile counters start at zero
    }
}

// Token tiles of the gate/up GEMM: the Q8_1 planes of each tile's tokens in the MMA's operand order.
// grid = (max tiles, kCtas), a CTA takes every kCtas-th group of 8 token slots of its tile, a warp 8 chunks of 16 bytes of the group's eight tokens at a time: read row by row
// (128 bytes in a row), turned in shared memory, written as the 8 x 16 bytes of one core-matrix row group.  Columns without a token are
// left as they are (nobody reads their sums).  Bound by L1 wavefronts: lanes that read the eight tokens side by side, as their stores want them,
// took 32 a load where a row takes 4 (8192 tokens x 8 of 2048 columns: 74 -> 55 us; 512 x 8: 14.9 -> 14.0, where the chain tile, pair, row is the time).
template <int kCtas>
__global__ void __launch_bounds__(256) gather_tiles_kernel(const int32_t* tiles, const int32_t* perm, const int8_t* x_q, int64_t x_q_stride,
                                                           const float* x_d, int x_d_stride, const uint8_t* x_q8, uint8_t* b_tiles,
                                                           int64_t b_col16_bytes, int H, int top_k, int shared_sums, int T) {
    griddep_wait();
    if (threadIdx.x == 0) griddep_launch();
    const int j = blockIdx.x;
    const int listed = __ldcg(tiles);
    int4 t;
    if (j < listed) t = __ldcg(reinterpret_cast<const int4*>(tiles + kTileHeader) + j);
    else {
        const int i = j - listed;   // a shared expert's tiles of 32 tokens
        if (!shared_sums || i * 32 >= T) return;
        t = make_int4(-1, i * 32, min(32, T - i * 32), __ldcg(tiles + 1) + 2 * i);
    }
    __shared__ uint4 s_turn[8][2][8 * 9];   // (a row of nine: no two lanes of a quarter warp on the same banks, either way)
    const int sl = threadIdx.x & 7, lane_ch = threadIdx.x >> 3, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool sums = t.x < 0 && shared_sums;   // a shared expert with minimums
    const int npad = sums ? 32 : tile_width(t.z), nch = H / 16;
    if ((int)blockIdx.y * 8 >= t.z) return;
    // the tokens of the CTA's groups: those whose rows this lane reads, and the one of the slot that it writes
    auto token = [&](int c) { return c >= t.z ? -1 : t.x < 0 ? t.y + c : __ldcg(perm + t.y + c) / top_k; };
    int rows[16 / kCtas][2], toks[16 / kCtas];
#pragma unroll
    for (int n = 0; n < 16 / kCtas; ++n) {
        const int c0 = (blockIdx.y + n * kCtas) * 8;
        rows[n][0] = token(c0 + (lane >> 3)); rows[n][1] = token(c0 + 4 + (lane >> 3)); toks[n] = token(c0 + sl);
    }
    uint8_t* base = b_tiles + (size_t)t.w * b_col16_bytes;
    // a shared expert with minimums: blocks in tree order, stages of four, each with the blocks' sums (the Q8_1 rows' second half) behind it
    auto place = [&](int b) { return sums ? operand_min_block(b, H / 32) : b; };
    auto block = [&](int b) { return base + (sums ? (size_t)(b >> 2) * (npad * 160) + (b & 3) * (npad * 36) : (size_t)b * (npad * 36)); };
#pragma unroll
    for (int n = 0; n < 16 / kCtas; ++n) {
        const int grp = blockIdx.y + n * kCtas, c = grp * 8 + sl, tok = toks[n];
        if (grp * 8 >= t.z) return;
        for (int g = warp * 8; g < nch; g += 128) {
            uint4 v[2][2];
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int ch = g + 64 * u + (lane & 7);
                    v[u][h] = ch < nch && rows[n][h] >= 0 ? __ldcg(reinterpret_cast<const uint4*>(x_q + (size_t)rows[n][h] * x_q_stride) + ch) : make_uint4(0u, 0u, 0u, 0u);
                }
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int h = 0; h < 2; ++h) s_turn[warp][u][((lane >> 3) + 4 * h) * 9 + (lane & 7)] = v[u][h];
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int i = 4 * h + (lane >> 3), ch = g + 64 * u + i;
                    if (ch < nch && tok >= 0) *reinterpret_cast<uint4*>(block(place(ch >> 1)) + (ch & 1) * (npad * 16) + grp * 128 + sl * 16) = s_turn[warp][u][sl * 9 + i];
                }
            __syncwarp();
        }
        if (tok >= 0)
            for (int b = lane_ch; b < H / 32; b += 32) {
                const int at = place(b);
                *reinterpret_cast<float*>(block(at) + npad * 32 + c * 4) = __ldcg(x_d + (size_t)tok * x_d_stride + b);
                if (sums) {
                    const uint32_t ds = __ldcg(reinterpret_cast<const uint32_t*>(x_q8 + ((size_t)tok * (H / 32) + b) * kQ81Bytes));
                    *reinterpret_cast<float*>(base + (size_t)(at >> 2) * (npad * 160) + npad * 144 + (at & 3) * (npad * 4) + c * 4) = h2f(ds >> 16);
                }
            }
    }
}

cudaError_t launch_build_tiles(const int32_t* offsets, const int32_t* perm, int32_t* tiles, int32_t* list, int E, int T, int has_shared, int gemm_min,
                               int shared_32, int widest, cudaStream_t stream) {
    return launch_pdl(build_tiles_kernel, dim3(1), 256, 0, stream, offsets, perm, tiles, list, E, T, has_shared, gemm_min, shared_32, widest);
}

cudaError_t launch_gather_tiles(const int32_t* tiles, const int32_t* perm, const int8_t* x_q, int64_t x_q_stride, const float* x_d,
                                int x_d_stride, const uint8_t* x_q8, uint8_t* b_tiles, int64_t b_col16_bytes, int H, int top_k, int n_tiles_max,
                                bool shared_sums, int T, cudaStream_t stream) {
    if (n_tiles_max <= 0) return cudaSuccess;
    // eight CTAs per tile rather than sixteen, most of which have nothing to do, up to four tiles per SM.  Prefill call, us, 16 / 8: 256 Q8_0 experts, skewed, 512
    // tokens 188.1 / 185.9, 1024: 305.0 / 302.0, 2048: 526.7 / 523.3, 8192 (over the line) 1876 / 1886; with four 189.9, 304.6, 523.9, 1892
    auto* kernel = n_tiles_max <= 4 * sm_count() ? gather_tiles_kernel<8> : gather_tiles_kernel<16>;
    return launch_pdl(kernel, dim3(n_tiles_max, n_tiles_max <= 4 * sm_count() ? 8 : 16), 256, 0, stream, tiles, perm, x_q, x_q_stride, x_d, x_d_stride, x_q8, b_tiles, b_col16_bytes,
                      H, top_k, shared_sums ? 1 : 0, T);
}

}  // namespace chimere
