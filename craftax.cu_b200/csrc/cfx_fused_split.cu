// Fused policy forward for batches that leave SMs idle when every 128-env tile has one SM (or pair of
// SMs) of its own: a tile is given to a cluster of S CTAs (2 or 4), each of which owns 1/S of the hidden
// units.  What a small batch costs is one tile's chain of dependent steps; here the chain is
// shorter: a CTA multiplies 64 NS instead of 256 encoder columns, one gate slice (NS = 1) instead of four a
// layer, and sixteen worker warps share the expansion and the cell of 1/S of the units.
//
//   records   the tile's records are contiguous: four bulk copies of 32 rows into shared memory.  A row is an odd
//             number of words, so thread-per-row reads have no bank conflicts.  (Tensor boxes of 80 bytes a
//             row cost more than the rest of the encoder.)  Every CTA of
//             the cluster expands the whole record into tensor memory, chunk kc by warpgroup kc % 4 (but the first ones by all: Cfg::kFirst)
//   encoder   A from tensor memory, N = 64 NS own units
//   layers    A from shared memory: the layer's input as K blocks of 64 units (128-byte swizzled operand
//             tiles, 16 KB).  A CTA writes its own K blocks and copies them to the other CTAs (bulk
//             copies shared memory -> shared memory of the cluster, counted on the receiver's
//             barrier), a quadrant of 32 rows = 4 KB at a time, as soon as its four warps are done
//   state     boxes of 128 rows x 32 units by tensor copies, updated in place and written back (a thread's own
//             64 bytes of a row, read and written by the threads, kept the load/store unit busy for 4,000 cycles a
//             layer and with it every barrier operation of the SM)
//             A CTA with two slices has those of its rank and of its rank + 2, so that the first K blocks of a layer's input are the
//             slices that are ready first: the next layer's products with them run under the cells of the second ones
//   heads     in the CTAs that sample, over all rows; the quadrants of rows are sampled in different CTAs
// The cluster works on one tile and exits, so every barrier but those of the rings is used once or once a
// layer.  The products of a row are accumulated in the order of cfx_fused.cu: same bits.
// Tiles of 32 rows (ONE), the smallest batches: a quadrant of TMEM lanes belongs to one SM scheduler, so one
// quadrant of rows would leave three schedulers idle.  The operand chunks go to shared memory instead, all
// sixteen warps at three of them at a time, and all multiplications are the weight-stationary ones of 32 rows: their columns are spread over the
// quadrants, so every warp has four of a slice's units, and they are shorter (an encoder step 29 cycles instead of 49,
// one of the gates 73 instead of 96).  A slice's zh and zg are one product of 128 columns and its zp one of 64; the weights' copies
// put the units of a quadrant together (1,024 envs h256x2 12.7 -> 11.6 us, against products of 128 rows with a copy of the layer
// input in every quadrant of tensor memory).  The layer input has two buffers there, beside the records.
// The records lie where the layer input and the state boxes are later: REC_FREE is complete when every CTA has expanded its
// records.  With one input buffer, it is overwritten when every CTA has done its multiplications of the layer (MMA_DONE,
// which a CTA's commit signals in all of them).
// Measured (us a step in a stream, fp16; the persistent kernel, one CTA pair per two tiles -> here): h256x2, 32 envs 20.6 -> 8.7,
// 256 21.0 -> 9.2, 1,024 21.5 -> 9.8, 2,048 21.7 -> 14.3, 4,000 22.3 -> 16.7, 8,192 22.7 -> 18.7; classic h256x3, 1,024 envs 28.9 -> 13.9, 4,000
// 29.7 -> 23.8, 8,192 30.2 -> 26.0.  Bound by the chain of dependent steps and the 1.3 us between one kernel's end and the next one's start.
// In clusters of two an encoder's weights are 14 pieces of 16 KB a CTA: with one lane issuing them, 500 cycles a slot, and one a
// slot of 24 KB, the multiplications waited for them, 10,200 cycles to the encoder's end at 8,192 envs; now 8,700, with the MMA warp waiting for
// the records' conversion.  8,192 envs h256x2: 20.00 us before, 19.94 with the slices in turn, 19.46 with the weight warp converged, 19.08 with the
// slots full, 18.91 with the first two chunks and the first slice of the encoder's output handed on at once.
#include "cfx_fused_split.h"

#include <type_traits>

namespace cfx {
namespace fused {
namespace split {

constexpr int kWorkerWarp0 = 4, kWorkerWarps = 16, kThreads = (kWorkerWarp0 + kWorkerWarps) * 32;
constexpr int kABlock = kTile * 128;                 // K block of the layer input: [128 rows][64 K]
constexpr int kWSlots = 4, kWSlot = kGateBlockBytes; // weight ring: one gate K block (24 KB) a slot
constexpr int kSlicePiece = kSliceUnits * 128;       // a slice's rows of an encoder weight block
constexpr int kMaxChunks = Gm<CFX_GAME_CLASSIC>::kEncChunks;
constexpr int kASlots = 12;                          // operand chunks in tensor memory; a multiple of the warpgroups
constexpr int kSSlots = 4, kSBox = kTile * 128, kQuadBox = 32 * 128;   // state ring: 128 rows x 32 units a slot, copied 32 rows at a time
constexpr int kFirstChunks = 4;   // see role_worker
constexpr uint32_t kColAexp = 0, kColAcc = 384, kColHead = 448;
__host__ __device__ constexpr uint32_t col_gate(int j) { return 192u * (uint32_t)j; }   // over the operand chunks, done by then

// Clusters of four, tiles of more than 32 rows: 96 registers a thread at launch, then 64 for the four warps that copy and multiply and
// 104 for the sixteen workers (us a step without and with that: 2,048 envs h256x2 15.04 and 14.86, 4,000 17.75 and 17.60, classic
// h256x3 2,048 26.2 and 21.9).  Not in tiles of 32 rows, which need fewer, not in cfx_fused.cu, whose MMA warp is slower with 64 (262,144 envs 406 ->
// 418), and not with two CTAs, whose workers have two slices each and then go through local memory more often (8,192 envs, the same pairs:
// h256x2 20.05 and 20.21, with a bf16 record 21.89 and 22.34, h256x3 with an fp32 record 29.05 and 30.29, bf16 29.60 and 31.00; h128x2 13.92 and 13.95).
constexpr int kLaunchRegs = 96, kRoleRegs = 64, kWorkerRegs = 104;
static_assert(kWorkerWarp0 * kRoleRegs + kWorkerWarps * kWorkerRegs <= (kWorkerWarp0 + kWorkerWarps) * kLaunchRegs, "registers");
template <int S, bool ONE> constexpr bool kShareRegs = S == 4 && !ONE;

constexpr int kQuadBlock = 32 * 128;                  // ONE: an operand chunk's block, [32 rows][64 K]
constexpr uint32_t kGateB = 4 * 2 * kWarpUnits * 128;   // ONE: zh and zg of a slice, behind them its zp
constexpr uint32_t kColP = 32;                        // ONE: columns of zh and zg in a quadrant, behind them zp

// ONE, full game: the twelve chunks of map bytes are converted three at a time, which are the blocks of a ring slot, by twelve warps with a
// quarter of a chunk each, the tail's four meanwhile by the other four, one to an SM scheduler.  The multiplications of a slot run under the
// conversion of the next one.  (A chunk a warp, and the multiplications behind all of them: the last chunk was there 1,500 cycles after the records, and
// the encoder done 2,400 later; now 3,200 after the records.  32 envs h256x2 9.42 -> 9.25 us, 512 10.0 -> 9.7, h128x2 8.65 -> 8.34.)
constexpr int kMapItems = 4, kMapWarps = 12;

template <int GAME, int HID, int S> struct Cfg {
    static constexpr int kKB = HID / 64;                        // K blocks of a layer's input
    static constexpr int kNS = HID / 64 / S;                    // gate slices of a CTA
    static constexpr int kUnits = 64 * kNS;                     // hidden units of a CTA
    static constexpr int kFirst = GAME == CFX_GAME_FULL && kNS == 1 ? kFirstChunks : 0;   // chunks that come one by one, in tiles of more than 32 rows
    // slice j of a CTA, which is also the K block that it makes of a layer's input
    static __host__ __device__ constexpr int slice(int rank, int j) { return rank + S * j; }
    // Its rows of an encoder weight block, one piece a slice.  A ring slot has three pieces, and the pieces lie one behind the other
    // from slot to slot, so that two of one block are one operand also where they are in two slots.
    static constexpr int kEncPieces = kNS * Gm<GAME>::kEncBlocks, kEncPerItem = kWSlot / kSlicePiece;
    static constexpr int kEncItems = (kEncPieces + kEncPerItem - 1) / kEncPerItem;
    static_assert(kEncPerItem * kSlicePiece == kWSlot && kWSlots * kEncPerItem % kNS == 0, "a block's pieces do not wrap around the ring");
    // ONE: how many warps bring the operand chunks of a ring slot
    static __device__ __forceinline__ int item_warps(int item) {
        if (GAME == CFX_GAME_FULL) return item < kMapItems ? kMapWarps : kWorkerWarps - kMapWarps;
        return max(1, min(kEncPerItem, Gm<GAME>::kEncBlocks - item * kEncPerItem));
    }
    static constexpr int kHeadHalf = Gm<GAME>::kHeadPair / 2 * 128;   // half of the head rows, one K block
    static constexpr int kHeadItems = kKB / 2;                  // two K blocks of the heads a slot
    static constexpr int kRowBytes = Gm<GAME>::kRecBytes, kQuadBytes = 32 * kRowBytes;
    static constexpr int kBoxes = 2 * kNS;                      // state boxes of a layer
    static constexpr int kOffS = kKB * kABlock, kASBytes = kOffS + kSSlots * kSBox;   // layer input, state; first the records
    static constexpr int kOffW = (kASBytes > 4 * kQuadBytes ? kASBytes : 4 * kQuadBytes + 1023) / 1024 * 1024;
    // ONE: operand chunks.  The classic game's 22 blocks
    // reach from the records over the layer input, the full game's 14 lie where the state boxes are later
    static constexpr int kOffX = GAME == CFX_GAME_FULL ? kOffS : 8192;
    static_assert(kOffX + Gm<GAME>::kEncBlocks * kQuadBlock <= kOffW && 32 * Gm<GAME>::kRecBytes <= kOffX, "operand chunks");
    // ONE: layer input l, K block kb, [32 rows][64 K]: two buffers in turn, so that nobody waits for the multiplications of
    // the layer before writing the next one's input; beside the records where there is room
    static constexpr bool kOneBeside = GAME == CFX_GAME_FULL && kOffS >= 32768 + kKB * 2 * kQuadBlock;
    static __device__ __forceinline__ uint32_t one_block(int l, int kb) {
        return (kOneBeside ? 32768 + kb * 2 * kQuadBlock : kb * kABlock) + (l & 1) * kQuadBlock;
    }
    // ONE, full game: the encoder's last two blocks, which the ring has no slots for, lie behind the operand chunks and, where there is room for one
    // alone, in the CTA's own blocks of the layer inputs, which it writes when the encoder is done
    template <bool ONE> static constexpr int ring_items() { return ONE && GAME == CFX_GAME_FULL ? kWSlots : kEncItems; }
    static_assert(kOffX + Gm<GAME>::kEncBlocks * kQuadBlock + (GAME == CFX_GAME_FULL ? kOneBeside ? 1 : 2 : 0) * kSlicePiece <= kOffW, "last blocks");
    static __device__ __forceinline__ uint32_t last_block(int blk, uint32_t rank) {
        constexpr uint32_t behind = kOffX + Gm<GAME>::kEncBlocks * kQuadBlock;
        return blk == kWSlots * kEncPerItem ? behind : (kOneBeside ? one_block(0, (int)rank) : behind + kSlicePiece);
    }
    static constexpr int kOffBias = kOffW + kWSlots * kWSlot;
    static constexpr int kOffBars = kOffBias + (kUnits + kHeadMax) * 4;
    static_assert(kNS >= 1 && kNS <= 2 && kUnits * S == HID &&
                      4 * kHeadHalf <= kWSlot && kQuadBytes % 16 == 0 &&
                      kRowBytes % 8 == 4, "shapes");
};

enum Bar {
    W_FULL = 0, W_LAST = W_FULL + kWSlots, W_EMPTY = W_LAST + 1, REC_FULL = W_EMPTY + kWSlots, REC_FREE = REC_FULL + 4,
    AEXP_FULL = REC_FREE + 1, AEXP_EMPTY = AEXP_FULL + kMaxChunks, ACC_FULL = AEXP_EMPTY + kASlots,
    S_FULL = ACC_FULL + 1, ST_READY = S_FULL + kSSlots, MMA_DONE = ST_READY + kSSlots,
    QUAD = MMA_DONE + 1, G_FULL = QUAD + 8,   // QUAD: [slice][quadrant]
    H_FULL = G_FULL + 2, A_KB = H_FULL + 1,
    // AEXP_FULL: four chunks each (ONE: of a ring slot).  Where the first kFirst chunks come by themselves (Cfg::kFirst) they have the last barriers of this
    // range, and those of four chunks that they would be part of are not used
    AEXP_FIRST = AEXP_FULL + kMaxChunks - kFirstChunks,
    // A_KB: [layer input][K block]; ONE: [layer input][0] for all of its blocks, but not for those of the heads' input
    NUM_BARS = A_KB + (kMaxLayers + 1) * 4
};
template <int GAME, int HID, int S> constexpr int smem_bytes() {
    return Cfg<GAME, HID, S>::kOffBars + NUM_BARS * 8 + 16 + 4 * kTile + 1024;   // misc, uniforms, alignment slack
}
static_assert(smem_bytes<CFX_GAME_FULL, 256, 2>() <= 232448 && smem_bytes<CFX_GAME_FULL, 128, 2>() <= 232448 && smem_bytes<CFX_GAME_FULL, 256, 4>() <= 232448 &&
                  smem_bytes<CFX_GAME_CLASSIC, 256, 4>() <= 232448, "shared memory");

constexpr uint32_t kSite = 0x40;   // wait-site codes: kSite + barrier

struct Smem {
    uint8_t* base;
    int off_bars;
    uint32_t bars;   // shared address of the barriers
    __device__ __forceinline__ uint32_t bar(int i) const { return bars + 8u * (uint32_t)i; }
    __device__ __forceinline__ uint32_t* tmem_base() const { return reinterpret_cast<uint32_t*>(base + off_bars + NUM_BARS * 8); }
    __device__ __forceinline__ float* uniforms() const { return reinterpret_cast<float*>(tmem_base() + 4); }   // of the rows that this CTA samples
    __device__ __forceinline__ volatile uint32_t* abort_flag() const { return tmem_base() + 1; }
};
// one lane waits (CFX_SWAIT1), or a whole warp (the MMA warp by polling alone)
#define CFX_SWAIT1(barid, parity) \
    if (!mbar_wait<false>(sm.bar(barid), (parity), sm.abort_flag(), kSite + (barid))) return
#define CFX_SWAIT(barid, parity) \
    if (!mbar_wait_warp<false>(sm.bar(barid), (parity), sm.abort_flag(), kSite + (barid))) return
#define CFX_SWAIT_SPIN(barid, parity) \
    if (!mbar_wait_warp<false, true>(sm.bar(barid), (parity), sm.abort_flag(), kSite + (barid))) return

#define CFX_SPROBE(name, barid, parity) CFX_PROBE(name, sm.bar(barid), (uint32_t)(parity))
#define CFX_SWAIT_PROBED(name, barid, parity)                                      \
    {                                                                              \
        uint32_t ready_;                                                           \
        CFX_PROBE_READ_ALL(name, ready_);                                              \
        if (ready_ == 0) CFX_SWAIT_SPIN(barid, parity);  \
    }

// arrives on the barrier in every CTA of the cluster when all MMAs issued so far are done
template <int S>
__device__ __forceinline__ void mma_commit_all(uint32_t bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
        "h"((uint16_t)((1u << S) - 1u))
        : "memory");
}

// The first min(S, quads) CTAs sample, one or two quadrants of rows each.  The others multiply no heads: nobody there
// would wait for the products, and a CTA must not leave while its multiplications run.
template <int S> __device__ __forceinline__ bool samples_rows(int quadrant, int quads, uint32_t rank) {
    return quadrant * min(S, quads) / quads == (int)rank;
}
template <int S, bool ONE> __device__ __forceinline__ bool has_heads(int quads, uint32_t rank) {
    if constexpr (ONE) return rank == 0;
    else if constexpr (S == 2) return true;   // a tile of more than 32 rows has two quadrants or more
    else return (int)rank < min(S, quads);
}

// ------------------------------------------------------------------ weights
// The operand image is the one that cfx_fused.cu uses.  A slice's rows of an encoder block are contiguous in it, and so is a
// gate K block.  The whole warp walks the ring, the next slot is probed before the copies into this one, and an elected lane issues.
template <int GAME, int HID, int S, bool ONE>
__device__ __forceinline__ void role_weights(const Smem& sm, const Params& P, uint32_t rank) {
    using C = Cfg<GAME, HID, S>;
    constexpr int kSlices = HID / 64;
    constexpr size_t enc_b = enc_bytes<GAME, HID>();
    const int gates = P.L * C::kNS * C::kKB;
    constexpr int kEnc = C::template ring_items<ONE>();
    const int items = kEnc + gates + (has_heads<S, ONE>(P.tile_rows / 32, rank) ? C::kHeadItems : 0);
    const uint32_t ring = smem_u32(sm.base + C::kOffW);
    for (int i = 0; i < items; i++) {
        const int slot = i % kWSlots, slot1 = (i + 1) % kWSlots;
        if (i >= kWSlots) {
            uint32_t ready;
            CFX_PROBE_READ_ALL(cfx_p_w, ready);
            if (ready == 0) CFX_SWAIT(W_EMPTY + slot, ((i / kWSlots) - 1) & 1);
        }
        if (i + 1 >= kWSlots) CFX_SPROBE(cfx_p_w, W_EMPTY + slot1, (((i + 1) / kWSlots) - 1) & 1);
        __syncwarp();
        if (!elect_one()) continue;
        const uint32_t dst = ring + slot * kWSlot, full = sm.bar(W_FULL + slot);
        if (i < kEnc) {
            const int pieces = min(C::kEncPerItem, C::kEncPieces - i * C::kEncPerItem);
            mbar_arrive_expect_tx(full, pieces * kSlicePiece);
            for (int q = 0; q < pieces; q++) {
                const int p = i * C::kEncPerItem + q, blk = p / C::kNS, slice = C::slice((int)rank, p % C::kNS);
                bulk_g2s(dst + q * kSlicePiece, P.image + (size_t)blk * Hd<HID>::kEncBlockBytes + (size_t)slice * kSlicePiece, kSlicePiece, full);
            }
            if (kEnc < C::kEncItems && i == kEnc - 1) {
                mbar_arrive_expect_tx(sm.bar(W_LAST), (C::kEncPieces - kEnc * C::kEncPerItem) * kSlicePiece);
                for (int blk = kEnc * C::kEncPerItem; blk < C::kEncPieces; blk++)
                    bulk_g2s(smem_u32(sm.base) + C::last_block(blk, rank), P.image + (size_t)blk * Hd<HID>::kEncBlockBytes + (size_t)rank * kSlicePiece, kSlicePiece, sm.bar(W_LAST));
            }
        } else if (i < kEnc + gates) {
            const int g = i - kEnc, kb = g % C::kKB, j = g / C::kKB % C::kNS, l = g / (C::kKB * C::kNS);
            const int blk = (l * kSlices + C::slice((int)rank, j)) * C::kKB + kb;
            mbar_arrive_expect_tx(full, kGateBlockBytes);
            const uint8_t* src = P.image + enc_b + (size_t)blk * kGateBlockBytes;
            if constexpr (ONE) {
                tensor_g2s_4d(dst, &P.gate_map[0], 0, 0, 0, 4 * blk, full);
                tensor_g2s_4d(dst + kGateB, &P.gate_map[1], 0, 0, 2, 4 * blk, full);
            } else {
                bulk_g2s(dst, src, kGateBlockBytes / 2, full);
                bulk_g2s(dst + kGateBlockBytes / 2, src + kGateBlockBytes / 2, kGateBlockBytes / 2, full);
            }
        } else {
            const int h = i - kEnc - gates;
            const uint8_t* src = P.image + enc_b + (size_t)P.L * kSlices * C::kKB * kGateBlockBytes;
            mbar_arrive_expect_tx(full, 4 * C::kHeadHalf);
#pragma unroll
            for (int b = 0; b < 2; b++)
#pragma unroll
                for (int half = 0; half < 2; half++)
                    bulk_g2s(dst + (2 * b + half) * C::kHeadHalf, src + (size_t)(half * C::kKB + 2 * h + b) * C::kHeadHalf, C::kHeadHalf, full);
        }
    }
}

// ------------------------------------------------------------------ MMA
// The whole warp walks through the steps and an elected lane issues: with the code uniform over the warp the compiler keeps
// descriptors in uniform registers (one lane alone in a branch: 2 to 6 % slower a step).  There is one tile, so every ring
// position is a compile-time constant and every descriptor one addition away from two bases: an MMA whose descriptor is
// computed takes ~150 cycles to issue, and 54 of them were two thirds of the encoder.  The barriers of the next step are
// probed before the current step's MMAs (CFX_PROBE), so that a probe's round trip runs under their issue.
template <typename T16, int GAME, int HID, int S>
__device__ __forceinline__ void role_mma(const Smem& sm, const Params& P, uint32_t tmem, uint32_t rank) {
    using C = Cfg<GAME, HID, S>;
    constexpr uint32_t fmt = Op16<T16>::kFmt;
    constexpr uint32_t idesc_enc = make_idesc(fmt, kTile, C::kUnits), idesc_gate = make_idesc(fmt, kTile, 3 * kSliceUnits),
                       idesc_head = make_idesc(fmt, kTile, Gm<GAME>::kHeadSingle);
    constexpr int kChunks = Gm<GAME>::kEncChunks, kGateItems = C::kNS * C::kKB;
    static_assert(kGateItems % kWSlots == 0 || kWSlots % kGateItems == 0, "a layer's first ring slot");
    const uint64_t wdesc = smem_desc_sw128(smem_u32(sm.base + C::kOffW)), adesc = smem_desc_sw128(smem_u32(sm.base));
    // ---- encoder
    auto aexp = [](int kc) { return kc < C::kFirst ? AEXP_FIRST + kc : AEXP_FULL + kc / 4; };
    static_assert(C::kFirst % 4 == 0 && C::kFirst <= kFirstChunks && (C::kFirst == 0 || AEXP_FULL + (kChunks + 3) / 4 <= AEXP_FIRST) && (kChunks + 3) / 4 <= kMaxChunks,
                  "a barrier for either");
    CFX_SPROBE(cfx_p_b, W_FULL, 0);
    CFX_SPROBE(cfx_p_a, aexp(0), 0);
#pragma unroll
    for (int kc = 0; kc < kChunks; kc++) {
        // block of 64 K columns, first of its 16-byte K pieces, K steps (see expand_full), last chunk of its block
        const bool full = GAME == CFX_GAME_FULL;
        const int blk = full && kc >= 12 ? (kc < 14 ? 12 : 13) : kc, first = full && kc >= 12 ? (kc == 13 ? 6 : (kc == 15 ? 2 : 0)) : 0;
        const int ks = full ? full_ksteps(kc) : (kc == kChunks - 1 ? 1 : 4);
        const bool starts = !(full && (kc == 13 || kc == 15)), ends = !(full && (kc == 12 || kc == 14));
        const int as = kc % kASlots, piece = blk * C::kNS;
        if (starts)
#pragma unroll
            for (int p = piece; p < piece + C::kNS; p++) {
                const int item = p / C::kEncPerItem;
                if (p % C::kEncPerItem != 0) continue;   // waited for with an earlier piece
                CFX_SWAIT_PROBED(cfx_p_b, W_FULL + item % kWSlots, (item / kWSlots) & 1);
                CFX_SPROBE(cfx_p_b, W_FULL + (item + 1) % kWSlots, ((item + 1) / kWSlots) & 1);
            }
        // (four chunks, one of each warpgroup, are there at the same time)
        if (kc % 4 == 0 || kc < C::kFirst) {
            CFX_SWAIT_PROBED(cfx_p_a, aexp(kc), 0);
            const int next = kc + 1 < C::kFirst ? kc + 1 : kc / 4 * 4 + 4;
            if (next < kChunks) CFX_SPROBE(cfx_p_a, aexp(next), 0);
        }
        tc_fence_after_sync();
        __syncwarp();
        const uint64_t bd = wdesc + (uint64_t)((piece % (kWSlots * C::kEncPerItem) * kSlicePiece >> 4) + first);
        const uint32_t a = tmem + kColAexp + as * 32;
        if (elect_one()) {
#pragma unroll
            for (int k = 0; k < ks; k++)
                mma_f16_ts(tmem + kColAcc, a + 8 * k, bd + 2 * k, idesc_enc, (kc | k) != 0 ? 1u : 0u);
            if (kc + kASlots < kChunks) mma_commit(sm.bar(AEXP_EMPTY + as));
            if (kc == kChunks - 1) mma_commit(sm.bar(ACC_FULL));
            if (ends)
#pragma unroll
                for (int p = piece; p < piece + C::kNS; p++)
                    if ((p + 1) % C::kEncPerItem == 0 || p == C::kEncPieces - 1) mma_commit(sm.bar(W_EMPTY + p / C::kEncPerItem % kWSlots));
        }
    }
    // ---- layers and heads (a loop over the layers: straight-line code for all of them would be fetched cold)
    uint32_t wpar = 0;   // parity bit of every ring slot
#pragma unroll
    for (int i = 0; i < C::kEncItems; i++) wpar ^= 1u << (i % kWSlots);
    // the ring slot of a layer's first item: the same for every layer where its items are whole rounds of the ring
    auto first_slot = [&](int l) { return kGateItems % kWSlots == 0 ? C::kEncItems % kWSlots : (C::kEncItems + l * kGateItems) % kWSlots; };
#pragma unroll 1
    for (int l = 0; l < P.L; l++) {
        const int slot0 = first_slot(l);
        CFX_SPROBE(cfx_p_a, A_KB + 4 * l, 0);
        // this CTA's own K block of slice 0 first: that slice's gate columns are free when its cells have read them (those of slice 1
        // when its own block is there, which is waited for with the others)
        CFX_SWAIT_SPIN(A_KB + 4 * l + C::slice((int)rank, 0), 0);
#pragma unroll
        for (int j = 0; j < C::kNS; j++) {
#pragma unroll
            for (int kb = 0; kb < C::kKB; kb++) {
                const int slot = (slot0 + j * C::kKB + kb) % kWSlots, slot1 = (slot + 1) % kWSlots;
                if (j == 0) {
                    CFX_SWAIT_PROBED(cfx_p_a, A_KB + 4 * l + kb, 0);
                    if (kb + 1 < C::kKB) CFX_SPROBE(cfx_p_a, A_KB + 4 * l + kb + 1, 0);
                }
                CFX_SWAIT_PROBED(cfx_p_b, W_FULL + slot, wpar >> slot & 1u);
                wpar ^= 1u << slot;
                CFX_SPROBE(cfx_p_b, W_FULL + slot1, wpar >> slot1 & 1u);
                tc_fence_after_sync();
                __syncwarp();
                const uint64_t bd = wdesc + (uint64_t)((slot * kWSlot) >> 4), ad = adesc + (uint64_t)((kb * kABlock) >> 4);
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < 4; ks++) mma_f16_ss(tmem + col_gate(j), ad + 2 * ks, bd + 2 * ks, idesc_gate, (kb | ks) != 0 ? 1u : 0u);
                    if (kb == C::kKB - 1) mma_commit(sm.bar(G_FULL + j));
                    if (j == C::kNS - 1 && kb == C::kKB - 1) mma_commit_all<S>(sm.bar(MMA_DONE));
                    mma_commit(sm.bar(W_EMPTY + slot));
                }
            }
        }
    }
    if (__builtin_expect(!has_heads<S, false>(P.tile_rows / 32, rank), 0)) {
        // no heads here: what is on its way to this CTA (the last layer's output) or was issued by it is only waited for
        for (int kb = 0; kb < C::kKB; kb++) CFX_SWAIT(A_KB + 4 * P.L + kb, 0);
        __syncwarp();
        if (elect_one()) mma_commit(sm.bar(H_FULL));
        CFX_SWAIT(H_FULL, 0);
        return;
    }
    const int slot0 = first_slot(P.L);
    CFX_SPROBE(cfx_p_a, A_KB + 4 * P.L, 0);
#pragma unroll
    for (int kb = 0; kb < C::kKB; kb++) {
        const int slot = (slot0 + kb / 2) % kWSlots, slot1 = (slot + 1) % kWSlots;
        CFX_SWAIT_PROBED(cfx_p_a, A_KB + 4 * P.L + kb, 0);
        if (kb + 1 < C::kKB) CFX_SPROBE(cfx_p_a, A_KB + 4 * P.L + kb + 1, 0);
        if (kb % 2 == 0) {
            CFX_SWAIT_PROBED(cfx_p_b, W_FULL + slot, wpar >> slot & 1u);
            CFX_SPROBE(cfx_p_b, W_FULL + slot1, wpar >> slot1 & 1u);
        }
        tc_fence_after_sync();
        __syncwarp();
        const uint64_t bd = wdesc + (uint64_t)((slot * kWSlot + (kb & 1) * 2 * C::kHeadHalf) >> 4), ad = adesc + (uint64_t)((kb * kABlock) >> 4);
        if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < 4; ks++) mma_f16_ss(tmem + kColHead, ad + 2 * ks, bd + 2 * ks, idesc_head, (kb | ks) != 0 ? 1u : 0u);
            if (kb == C::kKB - 1) mma_commit(sm.bar(H_FULL));
        }
    }
}

// ONE: a layer's weights are waited for while its input is on its way, and its input is one wait for all of its blocks, so that the 32 products of
// a layer are one run, as long as the issue of its products takes (the blocks come at about the same time; with a wait for each, and the weights' waits between
// them, 120 cycles a block).  The encoder's weights are waited for slot by slot: a CTA that starts where another one has ended has the first ones
// 400 cycles before the last.  The heads take their input block by block, as the first one is their CTA's own and there 900 cycles before the others (in one
// run 0.2 us slower).  us a step, h256x1 / x2 / x4 at 512 envs 7.92 / 9.76 / 13.45 -> 7.69 / 9.38 / 12.78, 32 envs h256x2 9.14 -> 8.74, 1,056 10.25 -> 9.97,
// h128x2 512 8.17 -> 7.93, classic h256x3 512 13.98 -> 13.49; of that 0.1 to 0.15 by the encoder's last blocks beside the ring (last_block), without
// which the first layer's last weights come late.
template <typename T16, int GAME, int HID, int S>
__device__ __forceinline__ void role_mma_one(const Smem& sm, const Params& P, uint32_t tmem, uint32_t rank) {
    using C = Cfg<GAME, HID, S>;
    constexpr uint32_t fmt = Op16<T16>::kFmt;
    // (M = 32 takes N = 64, 128 or 256)
    constexpr uint32_t idesc_64 = make_idesc(fmt, 32, kSliceUnits), idesc_hg = make_idesc(fmt, 32, 2 * kSliceUnits);
    constexpr int kBlocks = Gm<GAME>::kEncBlocks, kEnc = C::template ring_items<true>();
    static_assert(C::kEncItems <= kMaxChunks, "a barrier a ring slot");
    static_assert(C::kUnits == kSliceUnits && C::kKB <= kWSlots && C::kHeadItems <= kWSlots, "a layer's weights are in the ring at once");
    const uint64_t wdesc = smem_desc_sw128(smem_u32(sm.base + C::kOffW)), adesc = smem_desc_sw128(smem_u32(sm.base));
    const uint64_t xdesc = smem_desc_sw128(smem_u32(sm.base + C::kOffX));
    // ---- encoder
    CFX_SPROBE(cfx_p_b, W_FULL, 0);
    CFX_SPROBE(cfx_p_a, AEXP_FULL, 0);
#pragma unroll
    for (int item = 0; item < C::kEncItems; item++) {
        const int slot = item % kWSlots;
        CFX_SWAIT_PROBED(cfx_p_b, item < kEnc ? W_FULL + slot : W_LAST, item < kEnc ? (item / kWSlots) & 1 : 0);
        if (item + 1 < C::kEncItems) CFX_SPROBE(cfx_p_b, item + 1 < kEnc ? W_FULL + (item + 1) % kWSlots : W_LAST, item + 1 < kEnc ? ((item + 1) / kWSlots) & 1 : 0);
        CFX_SWAIT_PROBED(cfx_p_a, AEXP_FULL + item, 0);
        if (item + 1 < C::kEncItems) CFX_SPROBE(cfx_p_a, AEXP_FULL + item + 1, 0);
        tc_fence_after_sync();
        __syncwarp();
        if (elect_one()) {
#pragma unroll
            for (int b = 0; b < C::kEncPerItem; b++) {
                const int blk = item * C::kEncPerItem + b, last = kBlocks - 1;
                if (blk > last) break;
                const int ks = blk < last ? 4 : (GAME == CFX_GAME_FULL ? 2 : 1);
                const uint64_t bd = item < kEnc ? wdesc + (uint64_t)((slot * kWSlot + b * kSlicePiece) >> 4) : adesc + (uint64_t)(C::last_block(blk, rank) >> 4);
#pragma unroll
                for (int k = 0; k < ks; k++)
                    mma_f16_ws_ss(tmem + kColAcc, xdesc + (uint64_t)((blk * kQuadBlock) >> 4) + 2 * k, bd + 2 * k, idesc_64, (blk | k) != 0 ? 1u : 0u);
            }
            if (item == C::kEncItems - 1) mma_commit(sm.bar(ACC_FULL));
            if (item < kEnc) mma_commit(sm.bar(W_EMPTY + slot));
        }
    }
    // ---- layers (a loop: straight-line code for all of them would be fetched cold)
    uint32_t wpar = 0;   // parity bit of every ring slot
#pragma unroll
    for (int i = 0; i < kEnc; i++) wpar ^= 1u << (i % kWSlots);
    // the ring slot of a layer's first item: the same for every layer where its items are whole rounds of the ring
    auto first_slot = [&](int l) { return C::kKB % kWSlots == 0 ? kEnc % kWSlots : (kEnc + l * C::kKB) % kWSlots; };
#pragma unroll 1
    for (int l = 0; l < P.L; l++) {
        const int slot0 = first_slot(l);
#pragma unroll
        for (int kb = 0; kb < C::kKB; kb++) {
            const int slot = (slot0 + kb) % kWSlots;
            CFX_SWAIT_SPIN(W_FULL + slot, wpar >> slot & 1u);
            wpar ^= 1u << slot;
        }
        CFX_SWAIT_SPIN(A_KB + 4 * l, 0);
        tc_fence_after_sync();
        __syncwarp();
        if (elect_one()) {
#pragma unroll
            for (int kb = 0; kb < C::kKB; kb++) {
                const int slot = (slot0 + kb) % kWSlots;
                const uint64_t bd = wdesc + (uint64_t)((slot * kWSlot) >> 4), ad = adesc + (uint64_t)(C::one_block(l, kb) >> 4);
#pragma unroll
                for (int ks = 0; ks < 4; ks++) {
                    mma_f16_ws_ss(tmem + col_gate(0), ad + 2 * ks, bd + 2 * ks, idesc_hg, (kb | ks) != 0 ? 1u : 0u);
                    mma_f16_ws_ss(tmem + col_gate(0) + kColP, ad + 2 * ks, bd + (uint64_t)(kGateB >> 4) + 2 * ks, idesc_64, (kb | ks) != 0 ? 1u : 0u);
                }
                if (kb == C::kKB - 1) mma_commit(sm.bar(G_FULL));
                mma_commit(sm.bar(W_EMPTY + slot));
            }
        }
    }
    if (__builtin_expect(!has_heads<S, true>(1, rank), 0)) {
        // no heads here: what is on its way to this CTA (the last layer's output) or was issued by it is only waited for
        for (int kb = 0; kb < C::kKB; kb++) CFX_SWAIT(A_KB + 4 * P.L + kb, 0);
        __syncwarp();
        if (elect_one()) mma_commit(sm.bar(H_FULL));
        CFX_SWAIT(H_FULL, 0);
        return;
    }
    const int slot0 = first_slot(P.L);
#pragma unroll
    for (int i = 0; i < C::kHeadItems; i++) CFX_SWAIT_SPIN(W_FULL + (slot0 + i) % kWSlots, wpar >> (slot0 + i) % kWSlots & 1u);
    // (a block at a time: the first one is this CTA's own, which is there before the others)
    CFX_SPROBE(cfx_p_a, A_KB + 4 * P.L, 0);
#pragma unroll
    for (int kb = 0; kb < C::kKB; kb++) {
        CFX_SWAIT_PROBED(cfx_p_a, A_KB + 4 * P.L + kb, 0);
        if (kb + 1 < C::kKB) CFX_SPROBE(cfx_p_a, A_KB + 4 * P.L + kb + 1, 0);
        tc_fence_after_sync();
        __syncwarp();
        const int slot = (slot0 + kb / 2) % kWSlots;
        const uint64_t bd = wdesc + (uint64_t)((slot * kWSlot + (kb & 1) * 2 * C::kHeadHalf) >> 4), ad = adesc + (uint64_t)(C::one_block(P.L, kb) >> 4);
        if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < 4; ks++) mma_f16_ws_ss(tmem + kColHead, ad + 2 * ks, bd + 2 * ks, idesc_64, (kb | ks) != 0 ? 1u : 0u);
            if (kb == C::kKB - 1) mma_commit(sm.bar(H_FULL));
        }
    }
}

// ------------------------------------------------------------------ state
// One thread: box b of the tile (layer b / kBoxes, 32 units of all rows) uses slot b % kSSlots; a slot is loaded again when
// the box before has been read out of it.
template <int GAME, int HID, int S, bool ONE>
__device__ __forceinline__ void role_state(const Smem& sm, const Params& P, int row0, uint32_t rank) {
    using C = Cfg<GAME, HID, S>;
    const int boxes = P.L * C::kBoxes;
    const int quads = P.tile_rows / 32;
    auto slot_at = [&](int b) { return smem_u32(sm.base + C::kOffS + (b % kSSlots) * kSBox); };
    auto unit = [&](int b) { return C::slice((int)rank, b % C::kBoxes / 2) * kSliceUnits + b % 2 * 32; };
    auto load = [&](int b) {
        mbar_arrive_expect_tx(sm.bar(S_FULL + b % kSSlots), quads * kQuadBox);
        for (int q = 0; q < quads; q++)
            tensor_g2s_2d(slot_at(b) + q * kQuadBox, &P.state_map[b / C::kBoxes], unit(b), row0 + 32 * q, sm.bar(S_FULL + b % kSSlots));
    };
    if (!(ONE && C::kOneBeside)) CFX_SWAIT1(REC_FREE, 0);
    if (ONE) CFX_SWAIT1(ACC_FULL, 0);   // the operand chunks are used up
    for (int b = 0; b < kSSlots && b < boxes; b++) load(b);
    for (int b = 0; b < boxes; b++) {
        CFX_SWAIT1(ST_READY + b % kSSlots, (b / kSSlots) & 1);
        for (int q = 0; q < quads; q++) tensor_s2g_2d(&P.state_map[b / C::kBoxes], slot_at(b) + q * kQuadBox, unit(b), row0 + 32 * q);
        bulk_commit_group();
        if (b + kSSlots < boxes) {
            bulk_wait_group_read<0>();
            load(b + kSSlots);
        }
    }
    bulk_wait_group<0>();
}

// A part of the layer input that this CTA has made, to the CTA `d` ranks on: signalled on the barrier here, or copied and counted
// there.  (A warp for each: 1,024 envs 13.7 us with one lane issuing all copies, 13.6 so.)
template <int S>
__device__ __forceinline__ void hand_on(const Smem& sm, uint32_t offset, uint32_t bytes, int barrier, uint32_t rank, uint32_t d) {
    const uint32_t src = smem_u32(sm.base) + offset, bar = sm.bar(barrier), peer = (rank + d) % (uint32_t)S;
    if (d == 0) mbar_arrive(bar);
    else bulk_s2s(map_to_cta(src, peer), src, bytes, map_to_cta(bar, peer));
}

// ------------------------------------------------------------------ workers
// Sixteen warps: warp (quadrant, wg) owns TMEM lanes [32 quadrant, + 32) = those rows of the tile, converts a quarter of each of the first
// kFirst chunks, then chunks kFirst + wg, + 4, ..., and handles units [16 wg, 16 wg + 16) of every slice of the CTA.
template <typename T16, int GAME, int HID, int S, bool REC16>
__device__ __forceinline__ void role_worker(const Smem& sm, const Params& P, uint32_t tmem, int warp, int lane, int row0,
                                            uint32_t rank, Meetings& meet) {
    using Op = Op16<T16>;
    using C = Cfg<GAME, HID, S>;
    constexpr int kChunks = Gm<GAME>::kEncChunks, kA = Gm<GAME>::kA;
    const int quadrant = warp & 3, wg = (warp - kWorkerWarp0) >> 2, row = quadrant * 32 + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(quadrant * 32) << 16);
    const int env = row0 + row, quads = P.tile_rows / 32;
    if (quadrant >= quads) {   // (rows that nobody reads)
        meet.met = Meetings::kAll;
        return;
    }
    const bool valid = env < P.n;   // of a quadrant all rows or none (n is a multiple of 32)
    const float* bias = reinterpret_cast<const float*>(sm.base + C::kOffBias);
    const bool samples = samples_rows<S>(quadrant, quads, rank);
    const bool zero_state = valid && P.prev_terminals != nullptr && P.prev_terminals[env] != 0.0f;
    // (the flags are waited for here, under the records' way: with the ballot at its use, 8,192 envs took 21.8 us instead of 21.3)
    const uint32_t zero_rows = __ballot_sync(0xffffffffu, zero_state);
    if (valid && lane < P.L * C::kNS) {   // this warp's rows of the state, on their way to L2 while the records are expanded
        const float* q = P.state + ((size_t)(lane / C::kNS) * P.n + env - lane) * HID + C::slice((int)rank, lane % C::kNS) * kSliceUnits;
        for (int r = wg; r < 32; r += 4) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(q + (size_t)r * HID));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(q + (size_t)r * HID + 32));
        }
    }

    // ---- expand
    const uint8_t* rec = sm.base + row * C::kRowBytes;
    if (valid) CFX_SWAIT(REC_FULL + quadrant, 0);
    // a chunk is handed over after the next one is converted: the stores of the one drain meanwhile
    auto hand_over = [&](int kc) {
        tmem_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(sm.bar(AEXP_FULL + kc / 4));
    };
    // Full game, one slice a CTA: the first four chunks a quarter of each a warp, so that the encoder starts with the first one while the others are
    // converted.  (A chunk a warp, all four are there 1,100 cycles after the records.  us: 2,048 envs h256x2 14.37 -> 14.27, 4,224 with an fp32 record 18.50 -> 18.03,
    // 8,192 h128x2 13.39 -> 13.21.  With two slices a CTA the encoder's weights come too slowly for that to count: 8,192 h256x2 18.75 -> 18.68, with a bf16
    // record 6,400 h256x4 30.9 -> 31.2.)
    constexpr int kFirst = C::kFirst;
    if constexpr (kFirst > 0) {
        uint32_t bytes[4], regs[8];
        auto load = [&](int kc) {
#pragma unroll
            for (int q = 0; q < 4; q++) bytes[q] = valid ? *reinterpret_cast<const uint32_t*>(rec + 64 * kc + 16 * wg + 4 * q) : 0u;
        };
        auto there = [&](int kc) {
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(sm.bar(AEXP_FIRST + kc));
        };
        load(0);
#pragma unroll
        for (int kc = 0; kc < kFirst; kc++) {
#pragma unroll
            for (int q = 0; q < 4; q++) Op::bytes4(bytes[q], regs[2 * q], regs[2 * q + 1]);
            if (kc + 1 < kFirst) load(kc + 1);
            if (kc > 0) there(kc - 1);
            tmem_st8(lane_base + kColAexp + kc * 32 + 8 * wg, regs);
        }
        there(kFirst - 1);
    }
    for (int kc = kFirst + wg; kc < kChunks; kc += 4) {
        const int as = kc % kASlots;
        uint32_t regs[32];
        if (valid) {
            if constexpr (GAME == CFX_GAME_CLASSIC) expand_classic<Op>(rec, kc, regs);
            else expand_full<Op>(rec + 64 * kc, kc, regs);
        } else {
#pragma unroll
            for (int q = 0; q < 32; q++) regs[q] = 0u;
        }
        if (kc >= 12) hand_over(kc - 4);
        if (kc >= kASlots) {
            CFX_SWAIT(AEXP_EMPTY + as, ((kc / kASlots) - 1) & 1);
            tc_fence_after_sync();
        }
        uint32_t lo[16], hi[16];
#pragma unroll
        for (int q = 0; q < 16; q++) { lo[q] = regs[q]; hi[q] = regs[16 + q]; }
        tmem_st16(lane_base + kColAexp + as * 32, lo);
        tmem_st16(lane_base + kColAexp + as * 32 + 16, hi);
        if (kc < 8) hand_over(kc);   // (the first two at once: the MMA warp waits for them; 4,736 to 9,472 envs 0.3 to 0.5 % faster than with the first alone)
    }
    hand_over(wg + (kChunks - 1 - wg) / 4 * 4);
    __syncwarp();
    if (lane < S) mbar_arrive_cluster(map_to_cta(sm.bar(REC_FREE), (uint32_t)lane));
    // Hands this thread's 16 units of layer input l, slice j, on: into the own K block, and, once the quadrant's four
    // warps have done so, to the other CTAs, a warp of the quadrant for each.
    // (A barrier a slice: a warp may be one slice ahead of another, but not one layer.)
    auto send = [&](int l, int j, const uint32_t (&h)[8]) {
        const uint32_t kb = C::slice((int)rank, j), block = kb * kABlock;
        uint8_t* r = sm.base + block + (row >> 3) * 1024 + (row & 7) * 128;
#pragma unroll
        for (int q = 0; q < 2; q++)
            *reinterpret_cast<uint4*>(r + (((2 * wg + q) ^ (row & 7)) << 4)) = make_uint4(h[4 * q], h[4 * q + 1], h[4 * q + 2], h[4 * q + 3]);
        tc_fence_before_sync();
        fence_proxy_async_smem();
        __syncwarp();
        bool ok = true;
        if (lane == 0) {
            mbar_arrive(sm.bar(QUAD + 4 * j + quadrant));
            const uint32_t d = (uint32_t)(wg - quadrant) & 3u;
            if (d < (uint32_t)S) {
                ok = mbar_wait<false>(sm.bar(QUAD + 4 * j + quadrant), l & 1, sm.abort_flag(), kSite + QUAD);
                if (ok) hand_on<S>(sm, block + quadrant * (kABlock / 4), kABlock / 4, A_KB + 4 * l + (int)kb, rank, d);
            }
        }
        return __all_sync(0xffffffffu, ok);
    };

    // ---- encoder output + bias -> layer-0 input
    uint32_t x[C::kNS][8];   // this thread's units of the layer input, packed: operand and the cell's blend input
    CFX_SWAIT(REC_FREE, 0);   // (long complete when the accumulator is, and a wait takes 200 cycles all the same)
    CFX_SWAIT(ACC_FULL, 0);
    tc_fence_after_sync();
#pragma unroll
    for (int j = 0; j < C::kNS; j++) {
        uint32_t acc[16];
        tmem_ld16(lane_base + kColAcc + kSliceUnits * j + kWarpUnits * wg, acc);
        tmem_wait_ld();
        const float* b = bias + kSliceUnits * j + kWarpUnits * wg;
#pragma unroll
        for (int q = 0; q < 8; q++)
            x[j][q] = Op::pack(__uint_as_float(acc[2 * q]) + b[2 * q], __uint_as_float(acc[2 * q + 1]) + b[2 * q + 1]);
        if (!send(0, j, x[j])) return;
    }
    // The uniform of this row, which is there since the biases are (ACC_FULL).  In the classic game's kernel with one slice a CTA it is read ahead of the layers: so its cells
    // keep nothing in local memory (with an fp32 record, x3: 1,600 envs 22.4 -> 22.0 us, 3,200 26.4 -> 25.8).  In the others that costs registers (with a bf16
    // record 6,400 h256x2 20.0 -> 23.0; without one 8,192 classic x1 17.1 -> 17.2)
    constexpr bool kAhead = GAME == CFX_GAME_CLASSIC && C::kNS == 1;
    float u = 0.0f;
    if (kAhead && samples && wg == 0 && valid) u = *reinterpret_cast<volatile float*>(&sm.uniforms()[row]);
    // ---- layers
    for (int l = 0; l < P.L; l++) {
#pragma unroll
        for (int j = 0; j < C::kNS; j++) {
            const int box = l * C::kBoxes + 2 * j + (wg >> 1), slot = box % kSSlots;
            CFX_SWAIT(S_FULL + slot, (box / kSSlots) & 1);
            if (!REC16 && P.r_state != nullptr && valid)   // under the slice's MMAs
                write_r_state<4, HID>(P, sm.base + C::kOffS + slot * kSBox + quadrant * 4096, 4 * (wg & 1),
                                      ((size_t)l * P.n + row0 + 32 * quadrant) * HID + C::slice((int)rank, j) * kSliceUnits + wg * kWarpUnits,
                                      zero_rows, lane);
            CFX_SWAIT(G_FULL + j, l & 1);
            tc_fence_after_sync();
            uint32_t zh[16], zg[16], zp[16];
            tmem_ld16(lane_base + col_gate(j) + gate_row(0, kWarpUnits * wg), zh);
            tmem_ld16(lane_base + col_gate(j) + gate_row(1, kWarpUnits * wg), zg);
            tmem_ld16(lane_base + col_gate(j) + gate_row(2, kWarpUnits * wg), zp);
            tmem_wait_ld();
            uint8_t* sp = sm.base + C::kOffS + slot * kSBox + (row >> 3) * 1024 + (row & 7) * 128;
            auto piece = [&](int q) { return reinterpret_cast<float4*>(sp + (((4 * (wg & 1) + q) ^ (row & 7)) << 4)); };
            float rs[kWarpUnits / 2];   // REC16: the state record of this thread's units, packed
            // (half of the units at a time: with the state of all of them in registers a bf16 cell reads 22 words from local memory, so 4)
#pragma unroll
            for (int h = 0; h < kWarpUnits / 4; h += 2) {
                float4 st[2];
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    st[q] = *piece(h + q);
                    if (zero_state) st[q] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (REC16) {
                        rs[2 * (h + q)] = __uint_as_float(Op16<__nv_bfloat16>::pack(st[q].x, st[q].y));
                        rs[2 * (h + q) + 1] = __uint_as_float(Op16<__nv_bfloat16>::pack(st[q].z, st[q].w));
                    }
                }
                if (REC16 && h > 0 && valid)
                    st_global_v8(reinterpret_cast<float*>(reinterpret_cast<__nv_bfloat16*>(P.r_state) + ((size_t)l * P.n + env) * HID +
                                                          C::slice((int)rank, j) * kSliceUnits + wg * kWarpUnits), rs);
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const int i = 4 * (h + q);
                    const float2 x01 = Op::unpack(x[j][i / 2]), x23 = Op::unpack(x[j][i / 2 + 1]);
                    float h0, h1, h2, h3;
                    mingru_cell_pair(__uint_as_float(zh[i]), __uint_as_float(zh[i + 1]), __uint_as_float(zg[i]), __uint_as_float(zg[i + 1]),
                                     __uint_as_float(zp[i]), __uint_as_float(zp[i + 1]), st[q].x, st[q].y, x01.x, x01.y, st[q].x, st[q].y, h0, h1);
                    mingru_cell_pair(__uint_as_float(zh[i + 2]), __uint_as_float(zh[i + 3]), __uint_as_float(zg[i + 2]), __uint_as_float(zg[i + 3]),
                                     __uint_as_float(zp[i + 2]), __uint_as_float(zp[i + 3]), st[q].z, st[q].w, x23.x, x23.y, st[q].z, st[q].w, h2, h3);
                    x[j][i / 2] = Op::pack(h0, h1);
                    x[j][i / 2 + 1] = Op::pack(h2, h3);
                    *piece(h + q) = st[q];
                }
            }
            if (j == 0) CFX_SWAIT(MMA_DONE, l & 1);
            if (!send(l + 1, j, x[j])) return;
            if (lane == 0) mbar_arrive(sm.bar(ST_READY + slot));   // (send fenced the box as well)
        }
    }

    // ---- heads + sampler: the quadrant's four warps take a quarter of the exponentials each, then the first one draws
    if (samples) {
        constexpr int kHeadCols = (kA + 1 + 15) / 16 * 16, kPart = (kA + 3) / 4;
        CFX_SWAIT(H_FULL, 0);
        tc_fence_after_sync();
        uint32_t hv[kHeadCols];
#pragma unroll
        for (int b = 0; b < kHeadCols / 16; b++) {
            uint32_t t[16];
            tmem_ld16(lane_base + kColHead + 16 * b, t);
#pragma unroll
            for (int q = 0; q < 16; q++) hv[16 * b + q] = t[q];
        }
        tmem_wait_ld();
        const float* hb = bias + C::kUnits;
        float* p = reinterpret_cast<float*>(sm.base + C::kOffW) + row;   // [action][row]: all weights are used up
        float logits[kA];
#pragma unroll
        for (int a = 0; a < kA; a++) logits[a] = __uint_as_float(hv[a]) + hb[a];
        const float value = __uint_as_float(hv[kA]) + hb[kA];
        float m = logits[0];
#pragma unroll
        for (int a = 1; a < kA; a++) m = fmaxf(m, logits[a]);
#pragma unroll
        for (int a = 0; a < kA; a++)
            if (a / kPart == wg) p[a * kTile] = expf(logits[a] - m);
        if (wg == 1 && valid) write_logits<GAME>(P, env, logits, value);
        meet.sync(1 + quadrant, 128);
        if (wg == 0 && valid) {
            float pr[kA];
#pragma unroll
            for (int a = 0; a < kA; a++) pr[a] = p[a * kTile];
            float la = logits[0], total;
            const int act = draw_action<kA>(pr, kAhead ? u : sm.uniforms()[row], &total, [&](int a, bool beyond) { la = beyond ? logits[a + 1] : la; });
            write_action(P, env, act, la - m - logf(total), value);
        }
    }
    meet.met = Meetings::kAll;
}

// ONE: the sampler of 32 rows by all warps, lane = row in each: a warp brings four columns of the logits, their maximum and their
// exponentials to shared memory, then the first one sums, searches and draws, and the others write the logits.  All of it by
// one warp is the longest stretch of straight-line code in the chain of a step; with every warp taking the maximum of a
// whole row, and a sixteenth of the exponentials, 1,024 envs took 14.3 us instead of 13.8.
// `head`: tensor memory of this warp's lanes, `env`: of the lane; `uniforms`: of the rows
template <int GAME>
__device__ __forceinline__ void sample_one(const Params& P, float* s, uint32_t head, const float* bias, int w, int lane, int env, const float* uniforms,
                                           Meetings& meet) {
    constexpr int kA = Gm<GAME>::kA, kCols = 4, kWith = (kA + kCols) / kCols, kPitch = 33, W = kWorkerWarps;
    static_assert(kWith <= W && ((kA + 1) * kPitch + (kA + kWith) * 32) * 4 <= kWSlots * kWSlot, "scratch");
    float* p = s + (kA + 1) * kPitch + lane;   // logits [kA + 1][33], exponentials [kA][32], maxima [kWith][32]
    float* most = p + kA * 32;
    float l[kCols], m = -INFINITY;
    if (w < kWith) {
        uint32_t t[kCols];
        tmem_ld4(head, t);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < kCols; i++) {
            const int a = kCols * w + i;
            l[i] = a <= kA ? __uint_as_float(t[i]) + bias[a] : 0.0f;
            if (a <= kA) s[a * kPitch + lane] = l[i];
            if (a < kA) m = fmaxf(m, l[i]);
        }
        most[w * 32] = m;
    }
    meet.sync(1, 32 * W);
    if (w < kWith) {
#pragma unroll
        for (int i = 0; i < kWith; i++) m = fmaxf(m, most[i * 32]);
#pragma unroll
        for (int i = 0; i < kCols; i++)
            if (kCols * w + i < kA) p[(kCols * w + i) * 32] = expf(l[i] - m);
    }
    if (w != 0) {
        meet.arrive(1, 32 * W);
        if (P.logits_av != nullptr) {   // 32 rows, contiguous
            float* dst = P.logits_av + (size_t)(env - lane) * (kA + 1);
            for (int i = 32 * (w - 1) + lane; i < 32 * (kA + 1); i += 32 * (W - 1)) dst[i] = s[i % (kA + 1) * kPitch + i / (kA + 1)];
        }
    } else {
        meet.sync(1, 32 * W);
        float pr[kA], total;
#pragma unroll
        for (int a = 0; a < kA; a++) pr[a] = p[a * 32];
        const int act = draw_action<kA>(pr, uniforms[lane], &total, [](int, bool) {});
        write_action(P, env, act, s[act * kPitch + lane] - m - logf(total), s[kA * kPitch + lane]);
    }
}

// ONE: warp w = (quadrant, wg) converts its part of the record (kMapItems; classic game: chunk w and the one 16 further) and handles units
// [4 w, 4 w + 4) of the CTA's slice, which are in its quadrant of tensor memory; lane = row in all of it.
template <typename T16, int GAME, int HID, int S>
__device__ __forceinline__ void role_worker_one(const Smem& sm, const Params& P, uint32_t tmem, int warp, int lane, int row0,
                                                uint32_t rank, Meetings& meet) {
    using Op = Op16<T16>;
    using C = Cfg<GAME, HID, S>;
    constexpr int kChunks = Gm<GAME>::kEncChunks;
    constexpr bool kFull = GAME == CFX_GAME_FULL;
    const int quadrant = warp & 3, wg = (warp - kWorkerWarp0) >> 2, w = 4 * quadrant + wg, unit = 4 * w, swz = lane & 7;
    const uint32_t lane_base = tmem + ((uint32_t)(quadrant * 32) << 16);
    const int env = row0 + lane;
    const bool valid = env < P.n;   // all rows (n is a multiple of 32)
    const float* bias = reinterpret_cast<const float*>(sm.base + C::kOffBias);
    const bool zero_state = valid && P.prev_terminals != nullptr && P.prev_terminals[env] != 0.0f;
    if (lane < 2 * P.L)   // two rows of the state, on their way to L2 while the records are expanded
#pragma unroll
        for (int r = w; r < 32; r += kWorkerWarps)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(P.state + ((size_t)(lane >> 1) * P.n + row0 + r) * HID + rank * kSliceUnits + 32 * (lane & 1)));
    // 16-byte piece c of this lane's row of a 128-byte-swizzled block
    auto piece = [&](uint32_t block, int c) { return sm.base + block + (lane >> 3) * 1024 + swz * 128 + ((c ^ swz) << 4); };

    // ---- expand: K columns of a chunk go to the columns that its weight block has for them
    CFX_SWAIT(REC_FULL, 0);
    const uint8_t* rec = sm.base + lane * C::kRowBytes;
    auto operand = [&](int blk, int c, const uint32_t* r) {   // 16-byte piece c of this row in a block
        *reinterpret_cast<uint4*>(piece(C::kOffX + blk * kQuadBlock, c)) = make_uint4(r[0], r[1], r[2], r[3]);
    };
    auto converted = [&](int item) {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(sm.bar(AEXP_FULL + item));
    };
    if (kFull && wg < 3) {
        static_assert(C::kEncPerItem == 3 && kMapWarps == 3 * 4 && kMapItems * 3 == 12, "a warp a quarter of a chunk");
        // (a step's bytes are on their way while the one before is converted; all four steps' first: 0.05 to 0.1 us slower)
        uint32_t bytes[kMapItems][4];
        auto load = [&](int i) {
#pragma unroll
            for (int q = 0; q < 4; q++) bytes[i][q] = *reinterpret_cast<const uint32_t*>(rec + 64 * (3 * i + wg) + 16 * quadrant + 4 * q);
        };
        load(0);
#pragma unroll
        for (int i = 0; i < kMapItems; i++) {
            uint32_t regs[8];
            if (i + 1 < kMapItems) load(i + 1);
#pragma unroll
            for (int q = 0; q < 4; q++) Op::bytes4(bytes[i][q], regs[2 * q], regs[2 * q + 1]);
            operand(3 * i + wg, 2 * quadrant, regs);
            operand(3 * i + wg, 2 * quadrant + 1, regs + 4);
            converted(i);
        }
    } else {
        for (int kc = kFull ? 12 + quadrant : w; kc < kChunks; kc += kWorkerWarps) {
            uint32_t regs[32];
            if constexpr (kFull) expand_full<Op>(rec + 64 * kc, kc, regs);
            else expand_classic<Op>(rec, kc, regs);
            const int blk = kFull ? (kc < 14 ? 12 : 13) : kc;
            const int first = kFull ? (kc == 13 ? 6 : (kc == 15 ? 2 : 0)) : 0, pieces = 2 * (kFull ? full_ksteps(kc) : 4);
#pragma unroll
            for (int c = 0; c < 8; c++)
                if (c < pieces) operand(blk, first + c, regs + 4 * c);
            converted(blk / C::kEncPerItem);
        }
    }
    auto free_records = [&]() {
        __syncwarp();
        if (lane < S) mbar_arrive_cluster(map_to_cta(sm.bar(REC_FREE), (uint32_t)lane));
    };
    if (kFull && !C::kOneBeside) free_records();
    // Layer input l: the CTA's own K block is complete when all warps are here; then it goes to the other CTAs.
    auto send = [&](int l) {
        tc_fence_before_sync();
        fence_proxy_async_smem();
        __syncwarp();
        bool ok = true;
        if (lane == 0) {
            mbar_arrive(sm.bar(QUAD));
            if (w < S) {
                ok = mbar_wait<false>(sm.bar(QUAD), l & 1, sm.abort_flag(), kSite + QUAD);
                if (ok) hand_on<S>(sm, C::one_block(l, (int)rank), kQuadBlock, A_KB + 4 * l + (l == P.L ? (int)rank : 0), rank, (uint32_t)w);
            }
        }
        return __all_sync(0xffffffffu, ok);
    };
    // this thread's four units, bytes 8 (w & 1) of piece w / 2 of its row of the CTA's block
    auto xp = [&](int l) { return reinterpret_cast<uint2*>(piece(C::one_block(l, (int)rank), w >> 1) + 8 * (w & 1)); };

    // ---- encoder output + bias -> layer-0 input
    CFX_SWAIT(ACC_FULL, 0);
    tc_fence_after_sync();
    if (!kFull) free_records();
    if (!C::kOneBeside) CFX_SWAIT(REC_FREE, 0);
    uint2 x;   // this thread's units of the layer input, packed: operand and the cell's blend input
    {
        uint32_t acc[4];
        tmem_ld4(lane_base + kColAcc + 4 * wg, acc);
        tmem_wait_ld();
        const float* b = bias + unit;
        x = make_uint2(Op::pack(__uint_as_float(acc[0]) + b[0], __uint_as_float(acc[1]) + b[1]),
                       Op::pack(__uint_as_float(acc[2]) + b[2], __uint_as_float(acc[3]) + b[3]));
        *xp(0) = x;
    }
    if (!send(0)) return;

    // ---- layers
    for (int l = 0; l < P.L; l++) {
        const int box = l * C::kBoxes + (w >> 3), slot = box % kSSlots;
        CFX_SWAIT(S_FULL + slot, (box / kSSlots) & 1);
        float4* sp = reinterpret_cast<float4*>(piece(C::kOffS + slot * kSBox, w & 7));
        float4 st = *sp;
        if (zero_state) st = make_float4(0.f, 0.f, 0.f, 0.f);
        // optional BPTT record of the post-zero input state (craftax_full.cu:9370-9375)
        if (P.r_state != nullptr && valid) {
            const size_t at = ((size_t)l * P.n + env) * HID + rank * kSliceUnits + unit;
            if (P.r_state_bf16)
                *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(P.r_state) + at) =
                    make_uint2(Op16<__nv_bfloat16>::pack(st.x, st.y), Op16<__nv_bfloat16>::pack(st.z, st.w));
            else
                *reinterpret_cast<float4*>(P.r_state + at) = st;
        }
        CFX_SWAIT(G_FULL, l & 1);
        tc_fence_after_sync();
        uint32_t zh[4], zg[4], zp[4];
        tmem_ld4(lane_base + col_gate(0) + 4 * wg, zh);
        tmem_ld4(lane_base + col_gate(0) + kWarpUnits + 4 * wg, zg);
        tmem_ld4(lane_base + col_gate(0) + kColP + 4 * wg, zp);
        tmem_wait_ld();
        const float2 x01 = Op::unpack(x.x), x23 = Op::unpack(x.y);
        float h0, h1, h2, h3;
        mingru_cell_pair(__uint_as_float(zh[0]), __uint_as_float(zh[1]), __uint_as_float(zg[0]), __uint_as_float(zg[1]),
                         __uint_as_float(zp[0]), __uint_as_float(zp[1]), st.x, st.y, x01.x, x01.y, st.x, st.y, h0, h1);
        mingru_cell_pair(__uint_as_float(zh[2]), __uint_as_float(zh[3]), __uint_as_float(zg[2]), __uint_as_float(zg[3]),
                         __uint_as_float(zp[2]), __uint_as_float(zp[3]), st.z, st.w, x23.x, x23.y, st.z, st.w, h2, h3);
        x = make_uint2(Op::pack(h0, h1), Op::pack(h2, h3));
        *xp(l + 1) = x;
        if (!send(l + 1)) return;
        *sp = st;   // (behind what the next layer waits for: 512 envs h256x4 12.66 -> 12.56 us, 1,024 13.50 -> 13.39)
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(sm.bar(ST_READY + slot));
    }

    // ---- heads + sampler: all warps, each with the rows in its quadrant
    if (rank == 0) {
        CFX_SWAIT(H_FULL, 0);
        tc_fence_after_sync();
        if (valid) sample_one<GAME>(P, reinterpret_cast<float*>(sm.base + C::kOffW), lane_base + kColHead + 4 * wg, bias + C::kUnits, w, lane, env, sm.uniforms(), meet);
    }
    meet.met = Meetings::kAll;
}

// ------------------------------------------------------------------ kernel
template <typename T16, int GAME, int HID, int S, bool ONE, bool REC16>
__global__ void __launch_bounds__(kThreads, 1) k_policy_split(const __grid_constant__ Params P) {
    using C = Cfg<GAME, HID, S>;
    constexpr int kA = Gm<GAME>::kA;
    CFX_PROBE_DECL(cfx_p_a);
    CFX_PROBE_DECL(cfx_p_b);
    CFX_PROBE_DECL(cfx_p_w);
    extern __shared__ uint8_t smem_raw[];
    Smem sm;
    sm.base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    sm.off_bars = C::kOffBars;
    sm.bars = smem_u32(sm.base + C::kOffBars);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_ctarank();
    const int row0 = P.tile_begin * kTile + (int)blockIdx.x / S * P.tile_rows, quads = P.tile_rows / 32;
    launch_next_kernel();
    // Set-up: a CTA that starts where one of the kernel in front has just ended has none of it under that kernel, so it counts
    // (2,700 cycles with a few lanes setting all barriers up and everybody waiting for the cluster here).
    // A thread sets a barrier up.
    if (tid >= 32 * kWorkerWarp0) {
        const int i = tid - 32 * kWorkerWarp0;
        if (i < NUM_BARS) {
            uint32_t arrivals = 1, bytes = 0;
            if (i == REC_FREE) arrivals = ONE ? S * kWorkerWarps : S * 4 * quads;
            else if (i >= AEXP_FULL && i < AEXP_FULL + kMaxChunks)
                arrivals = ONE ? C::item_warps(i - AEXP_FULL)
                           : i >= AEXP_FIRST && C::kFirst > 0 ? 4 * quads : max(1, min(4, Gm<GAME>::kEncChunks - 4 * (i - AEXP_FULL))) * quads;
            else if (i == ACC_FULL) arrivals = 2;                          // the MMAs, and the biases are in place
            else if (i >= ST_READY && i < ST_READY + kSSlots) arrivals = ONE ? 8 : 2 * quads;
            else if (i == MMA_DONE) arrivals = S;
            else if (i >= QUAD && i < QUAD + 8) arrivals = ONE ? kWorkerWarps : 4;
            else if (i >= A_KB) {
                const int kb = (i - A_KB) % 4;
                if (ONE && (i - A_KB) / 4 < P.L) {   // one barrier for all blocks of a layer input: its own, and the bytes of the others
                    if (kb == 0) { arrivals = 2; bytes = (C::kKB - 1) * kQuadBlock; }
                } else if (kb < C::kKB && kb % S == (int)rank) arrivals = quads;
                else if (kb < C::kKB) bytes = quads * (kABlock / 4);       // a block of another CTA, counted by its bytes
            }
            mbar_init(sm.bar(i), arrivals);
            fence_mbar_init();
            if (bytes) mbar_arrive_expect_tx(sm.bar(i), bytes);
        }
        static_assert(NUM_BARS < 32 * kWorkerWarps, "a thread each");
        if (i == NUM_BARS) *sm.abort_flag() = 0;
        __syncwarp();
    } else if (warp == 1) {
        tmem_alloc(smem_u32(sm.tmem_base()), 512);
        tmem_relinquish();
    } else if (warp == 3) {
        if (lane == 0)
            for (int l = 0; l < P.L; l++) prefetch_tensormap(&P.state_map[l]);
        __syncwarp();
    }
    cluster_arrive_relaxed();   // waited for below, before the first access to another CTA
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *sm.tmem_base();

    // The operand image and the biases are only ever written by calls that wait for the device, so they may be
    // read while the kernel in front still runs; everything else waits for it.
    if (warp < kWorkerWarp0) {
        if constexpr (kShareRegs<S, ONE>) registers_dec<kRoleRegs>();
        if (warp == 0) {
            role_weights<GAME, HID, S, ONE>(sm, P, rank);
            __syncwarp();
            cluster_wait();
        } else if (warp == 1) {
            cluster_wait();
            if constexpr (ONE) role_mma_one<T16, GAME, HID, S>(sm, P, __shfl_sync(0xffffffffu, tmem, 0), rank);
            else role_mma<T16, GAME, HID, S>(sm, P, __shfl_sync(0xffffffffu, tmem, 0), rank);
        } else if (warp == 2) {
            // the tile's records, 32 rows a copy
            wait_for_previous_kernel();
            if (lane < quads && row0 + 32 * lane < P.n) {
                mbar_arrive_expect_tx(sm.bar(REC_FULL + lane), C::kQuadBytes);
                bulk_g2s(smem_u32(sm.base + lane * C::kQuadBytes), P.records + ((size_t)row0 + 32 * lane) * C::kRowBytes,
                         C::kQuadBytes, sm.bar(REC_FULL + lane));
            }
            for (int i = lane; i < C::kUnits + kA + 1; i += 32) {
                const int a = i - C::kUnits;
                reinterpret_cast<float*>(sm.base + C::kOffBias)[i] =
                    P.params[a < 0 ? P.off_b_enc + C::slice((int)rank, i / kSliceUnits) * kSliceUnits + i % kSliceUnits : (a < kA ? P.off_b_a + a : P.off_b_v)];
            }
            // The uniforms of the rows that this CTA samples, and the step counter, which the last CTA that has read it raises.  (By the workers that
            // sample, under the encoder's products, they were late in tiles of 32 rows, 512 envs h256x2 9.82 -> 9.72 us; in taller ones they cost registers:
            // 8,192 envs h256x2 with a bf16 record 21.46 -> 20.99, classic h256x3 26.4 -> 25.9, 4,736 h128x2 12.7 -> 12.2.)
            bool draws = false;
            const unsigned long long step0 = P.uniforms == nullptr && has_heads<S, ONE>(quads, rank) ? *P.step_ctr : 0ull;
            for (int q = 0; q < quads; q++)
                if (ONE ? rank == 0 : samples_rows<S>(q, quads, rank)) {
                    const int env = row0 + 32 * q + lane;   // (n is a multiple of 32)
                    draws = true;
                    if (env < P.n) sm.uniforms()[32 * q + lane] = P.uniforms != nullptr ? P.uniforms[env] : philox_uniform(P.seed, P.env_offset + (uint64_t)env, step0);
                }
            asm volatile("" ::"l"(step0));
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(sm.bar(ACC_FULL));
                if (draws && P.bump_step) done_with_step(P.step_ctr, P.done_ctr, P.done_blocks);
            }
            __syncwarp();
            cluster_wait();
        } else if (warp == 3) {
            wait_for_previous_kernel();
            cluster_wait();
            if (lane == 0) role_state<GAME, HID, S, ONE>(sm, P, row0, rank);
        }
    } else {
        if constexpr (kShareRegs<S, ONE>) registers_inc<kWorkerRegs>();
        wait_for_previous_kernel();
        cluster_wait();
        Meetings meet;
        if constexpr (ONE) role_worker_one<T16, GAME, HID, S>(sm, P, tmem, warp, lane, row0, rank, meet);
        else role_worker<T16, GAME, HID, S, REC16>(sm, P, tmem, warp, lane, row0, rank, meet);
        __syncwarp();
        if (__builtin_expect(meet.met != Meetings::kAll, 0)) {   // a wait gave up
            const int quadrant = warp & 3;
            if constexpr (ONE) {
                if (rank == 0 && row0 < P.n) meet.leave(1, 32 * kWorkerWarps, 2);
            } else {
                if (samples_rows<S>(quadrant, quads, rank)) meet.leave(1 + quadrant, 128, 1);
            }
        }
    }

    // common exit, also after a timed-out wait: no CTA leaves while another may still copy to it
    __syncwarp();
    tc_fence_before_sync();
    cluster_arrive_relaxed();
    cluster_wait();
    const uint32_t aborted = *sm.abort_flag();
    if (aborted != 0) {
        if (tid == 0) *reinterpret_cast<volatile uint32_t*>(P.status) = aborted | ((uint32_t)blockIdx.x << 8);
        for (int i = 0; i < 64; i++) __nanosleep(1000);   // time for copies in flight
        __syncthreads();
    }
    if (warp == 1) tmem_dealloc(tmem, 512);
}

static const void* kernel(int precision, int game, int H, int S, bool one, bool rec16, int* smem) {
    const bool h = precision == CFX_PREC_F16;
#define CFX_SPLIT(G, HID, SS)                                               \
    do {                                                                    \
        *smem = smem_bytes<G, HID, SS>();                                   \
        if constexpr (HID / 64 / SS == 1)                                   \
            if (one)                                                        \
                return h ? (const void*)k_policy_split<__half, G, HID, SS, true, false>          \
                         : (const void*)k_policy_split<__nv_bfloat16, G, HID, SS, true, false>;  \
        if constexpr (G == CFX_GAME_FULL && HID == 256)                     \
            if (rec16)                                                      \
                return h ? (const void*)k_policy_split<__half, G, HID, SS, false, true>          \
                         : (const void*)k_policy_split<__nv_bfloat16, G, HID, SS, false, true>;  \
        return h ? (const void*)k_policy_split<__half, G, HID, SS, false, false>          \
                 : (const void*)k_policy_split<__nv_bfloat16, G, HID, SS, false, false>;  \
    } while (0)
    if (game == CFX_GAME_CLASSIC) {
        if (S == 4) CFX_SPLIT(CFX_GAME_CLASSIC, 256, 4);
        CFX_SPLIT(CFX_GAME_CLASSIC, 256, 2);
    }
    if (H == 128) CFX_SPLIT(CFX_GAME_FULL, 128, 2);
    if (S == 4) CFX_SPLIT(CFX_GAME_FULL, 256, 4);
    CFX_SPLIT(CFX_GAME_FULL, 256, 2);
#undef CFX_SPLIT
}

static cudaLaunchConfig_t config(cudaLaunchAttribute (&at)[2], int blocks, int S, int smem, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)S; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // see wait_for_previous_kernel
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return cfg;
}

}  // namespace split

int split_prepare(int precision, int game, int H, int S, int sm_count, int* max_clusters) {
    *max_clusters = 0;
    if (H / 64 / S < 1) return CFX_OK;
    int smem = 0;
    const void* k = split::kernel(precision, game, H, S, true, false, &smem);
    CFX_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    for (int rec16 = 1; rec16 >= 0; rec16--) {
        k = split::kernel(precision, game, H, S, false, rec16 != 0, &smem);
        CFX_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        cudaFuncAttributes attr;
        CFX_CUDA(cudaFuncGetAttributes(&attr, k));
        // Built with fewer registers than its warps share out, they would wait for some that do not exist: such a build does without
        // this kernel, and cfx_fused.cu's takes every batch.
        if (S == 4 && attr.numRegs < split::kLaunchRegs) return CFX_OK;
    }
    cudaLaunchAttribute at[2];
    cudaLaunchConfig_t cfg = split::config(at, sm_count / S * S, S, smem, nullptr);
    cfg.numAttrs = 1;
    int nc = 0;
    if (cudaOccupancyMaxActiveClusters(&nc, k, &cfg) == cudaSuccess) *max_clusters = nc;
    else cudaGetLastError();
    return CFX_OK;
}

int split_launch(int precision, int game, int H, int S, int tiles, const Params& P, cudaStream_t st) {
    int smem = 0;
    const void* k = split::kernel(precision, game, H, S, P.tile_rows == 32, record_by_rows(P), &smem);
    cudaLaunchAttribute at[2];
    cudaLaunchConfig_t cfg = split::config(at, tiles * S, S, smem, st);
    void* args[1] = {(void*)&P};
    CFX_CUDA(cudaLaunchKernelExC(&cfg, k, args));
    return CFX_OK;
}

}  // namespace fused
}  // namespace cfx
