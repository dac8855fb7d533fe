// Fused policy forward for sm_100a: one persistent kernel runs, per 128-env tile,
//   compact records (bulk copies) -> fp16/bf16 operand rows written straight into tensor
//   memory -> encoder MMA -> MinGRU layers (gate MMA + cell epilogue, activations kept in
//   tensor memory as the next layer's A operand) -> actor/value MMA -> categorical sample.
// HBM traffic is the record, the fp32 recurrent state (read + written through TMA) and the
// outputs; weights stream from L2 through a shared-memory ring as pre-swizzled images.
//
// Replaces, inside cu_rollout_step (craftax_full.cu:12022-12087): k_expand_obs (:10028),
// the encoder GEMM + k_add_bias (:11954-11962), cu_gru_chain (:11978-12014: gate GEMM +
// k_mingru_epi_fwd :9350), the head GEMM (:12040-12045) and k_value_sample (:9714).
//
// Tile-level dataflow (M = 128 envs = the 128 TMEM lanes; the worker thread that owns TMEM lane
// r owns env row r of the tile in every phase):
//   TMEM columns   gate phase: A0 [0,128) A1 [128,256) (layer inputs, 16-bit packed, ping-pong)
//                              G [256,448) (gate accumulators of one 64-unit slice, zh|zg|zp of either
//                              half: while one half is multiplied, the workers take the other
//                              one's to registers, which frees it)  HEAD [448,512)
//                  encoder phase: operand-chunk ring [0,256) (8 x 32 columns), accumulator
//                              [256,512)
//   shared memory  weight ring | data area: the tile's records, then its state boxes | biases, barriers: see Cfg
//   warps          0 weight loads, 1 MMA issue + TMEM alloc, 2 records and state box loads (one
//                  thread), 3 state box stores (one thread), 4..19 workers in four groups of 128 rows (expand, cell; the
//                  first group samples)
//   launch modes   clusters of two CTAs sharing 256-row MMAs (PAIR, the default) or one CTA per
//                  tile; full game or classic game (GAME): see Cfg and Gm
//   hidden size    256 (the figures in this comment) or 128 (HID): two gate slices of two K
//                  blocks per layer, A0 / A1 of 64 columns, encoder accumulator N = 128: see Hd
// What bounds it: in long runs the board's power limit (1,000 W).  262,144 envs h256x2, 14 tiles a CTA, by the SM's clock and the global
// timer read in the kernel: in a long run 455,000 cycles in 394 us, 1.16 GHz (410 us a step; nvidia-smi reads 1.16 to 1.31 GHz
// meanwhile), in a burst of 20 launches 467,000 in 338 us, 1.38 GHz (346 us a step).  A CTA's first tile takes 41,000 cycles, the
// others 31,700, the last 30,800.  With eight worker warps, record boxes through a ring and one gate accumulator a tile took 39,900 and a
// step 415 us: that was 1.35 GHz, so fewer cycles come back as time only in part.  Without the MMAs a step takes 283 us at 1,965 MHz.
// Of a tile (33,700 cycles with the marks of a timeline): encoder 11,800, of which 2,300 until the last records are there
// and converted, 2,300 to the first gate accumulator, 2,300 a slice (1,540 of SFU and of tensor pipe), heads.  96 registers a thread,
// and 68 / 60 bytes of spill stores / loads (pairs, full game, hidden 256).  What mattered, all of it seen
// in clock64 timelines and rates of single instructions:
//   * a TMA store runs at 32 B a cycle, the SM's rate of writing, and copies queue behind it: 16 KB of state are 512
//     cycles.  Written by the workers instead (8 rows x 64 B an instruction) they held up the cells (262,144 envs 359 against 346 us);
//   * software prefetches to L2 of all that the next layer and tile load went through the same queue: 354 against 342 us;
//     of the records whose slots come free last they help (349 against 346);
//   * a round of (wait, arrive.expect_tx, copy) takes a lone thread 500 to 750 cycles, a converged warp with an elected lane 250;
//   * the tensor pipe queues four to five MMAs, and an MMA takes 33 cycles to issue: one wait and one commit per sixteen.
#include "cfx_fused_common.cuh"
#include "cfx_fused_split.h"

#include <algorithm>

namespace cfx {
namespace fused {

constexpr int kNBMax = 4;        // weight ring slots (one stage each): see Cfg
constexpr int kNS = 8, kSSlot = 16384;   // data slots: a state box or the records of 16 rows each
constexpr int kAexpSlots = 8;
constexpr int kKBlocksMax = 4;
constexpr int kHalfRows = 3 * kHalfUnits;   // gate columns of half a slice

// Barriers are waited on by phase parity, which is only sound while the waiter can never be
// two phases off.  So every slot of a ring has ONE filling thread, and every consumer sees every phase of
// the slots that it uses: a state box belongs to the two worker groups of its half of a slice and its slot is filled again when
// both are done with it; the weight ring has one consumer.  The operand slots in tensor memory are shared
// by the groups; there the order is carried by the commits, which come in the order of the chunks, and from one tile
// to the next by H_FULL, which all of them have passed.

// TMEM columns
constexpr uint32_t kColA0 = 0, kColA1 = 128, kColG = 256, kColHead = 448;
constexpr uint32_t kColAexp = 0, kColAcc = 256;

enum Bar {
    B_FULL = 0, B_EMPTY = B_FULL + kNBMax, S_FULL = B_EMPTY + kNBMax, S_FREE = S_FULL + kNS,
    ST_READY = S_FREE + kNS, REC_FULL = ST_READY + kNS, REC_FREE = REC_FULL + 4,
    AEXP_FULL = REC_FREE + 4, AEXP_EMPTY = AEXP_FULL + kAexpSlots,
    ACC_FULL = AEXP_EMPTY + kAexpSlots, A_KB = ACC_FULL + 1, G_FULL = A_KB + kKBlocksMax,
    G_EMPTY = G_FULL + 2, H_FULL = G_EMPTY + 2, H_EMPTY = H_FULL + 1, ACC_READ = H_EMPTY + 1, NUM_BARS = ACC_READ + 1
};

// Shared memory map (offsets from a 1024-byte aligned base) and the shapes that depend on the
// launch mode.
//  weight ring, a CTA pair (cta_group::2: every CTA stages half of the rows): four stages of 24 KB, an encoder block of 256
//    units or two of 128, or half a gate slice with all K blocks;
//  weight ring, one CTA per tile: a gate stage has two K blocks of half a slice (24 KB).  Hidden 256: four stages of 24 KB, and the
//    encoder blocks (32 KB), which lie one behind the other in the image, are cut every 192 rows.  Hidden 128: three of 32 KB.  us a
//    step, 131,072 envs h256x1, h256x3, h128x3, with two stages of 48 KB 162, 321, 157, three of 32 KB 152, 320, 139, four
//    of 24 KB with encoder blocks in halves 161, 308, 145, as it is 145, 294, 139: a stage's way from L2 takes about as long as the
//    products of two, so it is the number of full stages that counts;
//  data area: 8 x 16 KB.  First the tile's records, 16 rows a slot (the classic game's all in slots 0 and 1), then the state boxes
//    of the layers.  A slot's records of the next tile are fetched as soon as the last layer's box has left it: REC_FREE and
//    S_FREE order the two uses.
template <bool PAIR, int GAME, int HID> struct Cfg {
    static constexpr int kH = HID, kStateItems = Hd<HID>::kStateItems;
    static constexpr bool kCut = !PAIR && HID == 256;        // encoder stages of 192 rows: a block of 256 takes parts of two
    static constexpr int kNB = PAIR || kCut ? 4 : 3;
    static constexpr int kBSlot = PAIR || kCut ? 24576 : 32768;
    static constexpr int kEncPer = 256 / HID;                // encoder blocks of a stage that holds whole ones
    static constexpr int kEncRows = PAIR ? HID / 2 : HID;    // rows of a block that a CTA stages
    static constexpr int kCutRows = 192, kCutUnit = HID - kCutRows;   // three blocks are four stages
    static constexpr int kGateRows = PAIR ? kHalfRows / 2 : kHalfRows;
    static constexpr int kGateKb = PAIR ? Hd<HID>::kKBlocks : 2;   // K blocks of a gate stage
    static constexpr int kEncStages = kCut ? (Gm<GAME>::kEncBlocks * HID + kCutRows - 1) / kCutRows : Gm<GAME>::kEncBlocks / kEncPer;
    static constexpr int kLayerStages = 2 * Hd<HID>::kSlices * (Hd<HID>::kKBlocks / kGateKb);
    static constexpr int kHeadRows = PAIR ? Gm<GAME>::kHeadPair : Gm<GAME>::kHeadSingle;   // N of the head MMA
    static constexpr int kHeadKbBytes = (PAIR ? kHeadRows / 2 : kHeadRows) * 128;   // one K block of the head rows a CTA stages
    static constexpr int kM = PAIR ? 256 : 128;
    // State boxes that are loaded as soon as their slots are free of records.  The slots come free at about the same time, and copies
    // queue in order: with eight boxes (128 KB from memory) in front of them the last weight stages of the encoder came 2,500 cycles late.  The others
    // are loaded when the encoder is done.  us a step in long runs, all boxes at once and so: h256x2 18,944 envs 29.4 and 29.5, 37,888 63.7 and 62.1, 131,104
    // 210.7 and 207.5; h256x3 65,536 147.3 and 146.0; h128x2 131,104 112.6 and 111.1; within 0.6 % of each other above.
    // All at once where the state is recorded ahead of the cells (not REC16: h256x2 16,416 envs 29.5 and 29.2), and in the classic game, whose records
    // leave six of the slots alone (classic h256x3, at once and so: 9,504 envs 31.66 and 31.91, 1,048,576 2,192 and 2,197).
    static constexpr int kEarlyBoxes = HID == 256 ? 1 : 4;
    // records: rows of one copy, slots that hold them, where row r of the tile begins in the data area.  Full game: 16 rows a
    // slot, the odd slots 64 bytes on, so that a warp's 32 rows start in 32 banks
    static constexpr int kRecBytes = Gm<GAME>::kRecBytes, kRecRows = GAME == CFX_GAME_FULL ? 16 : kTile;
    static constexpr int kRecSlots = GAME == CFX_GAME_FULL ? 8 : 2, kRecCopies = kTile / kRecRows;
    static __device__ __forceinline__ int rec_offset(int r) {
        return GAME == CFX_GAME_FULL ? r / kRecRows * kSSlot + (r / kRecRows & 1) * 64 + r % kRecRows * kRecBytes : r * kRecBytes;
    }
    static constexpr int kOffB = 0;
    static constexpr int kOffS = kOffB + kNB * kBSlot;
    static constexpr int kOffBias = kOffS + kNS * kSSlot;      // b_enc fp32, b_av fp32
    static constexpr int kOffBars = kOffBias + (kH + kHeadMax) * 4;
    static constexpr int kOffMisc = kOffBars + NUM_BARS * 8;  // tmem base, abort flag
    static constexpr int kSmemBytes = kOffMisc + 16 + 1024;   // + alignment slack
    static_assert(kNB <= kNBMax && kSmemBytes <= 232448 && kHeadRows <= kHeadMax && kRecSlots <= kNS &&
                      64 + kRecRows * kRecBytes <= kRecSlots / kRecCopies * kSSlot && kRecRows * kRecBytes % 16 == 0 && kNS % kStateItems == 0 &&
                      Gm<GAME>::kEncBlocks % kEncPer == 0 && (kCut ? kCutRows : kEncPer * kEncRows) * 128 <= kBSlot && kGateKb * kGateRows * 128 <= kBSlot &&
                      Hd<HID>::kKBlocks * kHeadKbBytes <= kBSlot && kGateRows % 8 == 0, "layout");
};

constexpr int kWorkerWarp0 = 4, kGroups = 4, kWorkerWarps = 4 * kGroups, kNumWarps = kWorkerWarp0 + kWorkerWarps, kThreads = kNumWarps * 32;
static_assert(kWarpUnits * kGroups == kSliceUnits, "a group of four warps has 16 units of a slice");

// wait-site codes recorded in the status word when a bounded wait gives up
enum WaitCode : uint32_t {
    W_B_EMPTY = 1, W_B_FULL, W_REC_FULL, W_REC_FREE, W_S_FULL, W_S_FREE, W_ST_READY, W_AEXP_EMPTY,
    W_AEXP_FULL, W_ACC_FULL, W_A_KB, W_G_FULL, W_G_EMPTY, W_H_FULL, W_H_EMPTY, W_ACC_READ
};

// ------------------------------------------------------------------ weight image
template <typename T16>
__device__ inline T16 to16(float v);
template <>
__device__ inline __half to16<__half>(float v) {
    return __float2half_rn(fminf(fmaxf(v, -65504.0f), 65504.0f));
}
template <>
__device__ inline __nv_bfloat16 to16<__nv_bfloat16>(float v) {
    return __float2bfloat16_rn(v);
}

// One thread per 16-bit element of the image (layout: cfx_fused_common.cuh).
template <typename T16, int GAME, int HID>
__global__ void k_pack_image(const float* __restrict__ params, uint8_t* __restrict__ image, int L,
                             size_t off_w_gru, size_t off_w_a, size_t off_w_v, int pair) {
    CFX_DIMS(HID);
    constexpr int kA = Gm<GAME>::kA, kEncBlockBytes = Hd<HID>::kEncBlockBytes;
    const size_t total = image_bytes<GAME, HID>(L) / 2;
    size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const size_t byte = idx * 2, enc_b = enc_bytes<GAME, HID>();
    const size_t gate_bytes = (size_t)L * kSlices * kKBlocks * kGateBlockBytes;
    float v = 0.0f;
    int row, c;
    uint8_t* block;
    if (byte < enc_b) {
        const int blk = (int)(byte / kEncBlockBytes), e = (int)(byte % kEncBlockBytes / 2);
        row = e / 64; c = e % 64;
        block = image + (size_t)blk * kEncBlockBytes;
        const int f = enc_feature<GAME>(blk, c);
        if (f >= 0) v = params[(size_t)f * kH + row];
    } else if (byte < enc_b + gate_bytes) {
        const size_t b = byte - enc_b;
        const int blk = (int)(b / kGateBlockBytes), e = (int)(b % kGateBlockBytes / 2);
        const int kb = blk % kKBlocks, j = blk / kKBlocks % kSlices, l = blk / (kKBlocks * kSlices);
        row = e / 64; c = e % 64;
        block = image + enc_b + (size_t)blk * kGateBlockBytes;
        const int gate = row / kWarpUnits % 3, unit = j * kSliceUnits + row / (3 * kWarpUnits) * kWarpUnits + row % kWarpUnits;
        // gate weights are stored halved: the accumulator then holds z / 2, the argument of the
        // cell's tanh (a power-of-two scale is exact for every weight above the subnormal range)
        v = 0.5f * params[off_w_gru + ((size_t)l * 3 * kH + gate * kH + unit) * kH + kb * 64 + c];
    } else {
        // head.  One CTA per tile: [K block][rows][64 K].  CTA pairs: CTA r stages head rows
        // [r rows/2, (r + 1) rows/2): [r][K block][rows / 2][64 K].
        const size_t b = byte - enc_b - gate_bytes;
        if (b >= (size_t)head_bytes<GAME, HID>(pair != 0)) return;
        const int rows = pair ? Gm<GAME>::kHeadPair / 2 : Gm<GAME>::kHeadSingle;   // rows of one block
        const int blk_bytes = rows * 128;
        const int blk = (int)(b / blk_bytes), e = (int)((b % blk_bytes) / 2);
        const int r = pair ? blk / kKBlocks : 0, kb = blk % kKBlocks;
        row = e / 64; c = e % 64;
        block = image + enc_b + gate_bytes + (size_t)blk * blk_bytes;
        const int grow = rows * r + row;
        if (grow < kA) v = params[off_w_a + (size_t)grow * kH + kb * 64 + c];
        else if (grow == kA) v = params[off_w_v + kb * 64 + c];
    }
    *reinterpret_cast<T16*>(block + sw128_off((uint32_t)row, (uint32_t)c * 2)) = to16<T16>(v);
}

struct Smem {
    uint8_t* base;
    int off_s, off_bias, off_misc;
    uint32_t bars;   // shared address of the barriers
    template <bool PAIR, int GAME, int HID> __device__ __forceinline__ void layout() {
        using C = Cfg<PAIR, GAME, HID>;
        off_s = C::kOffS; off_bias = C::kOffBias; bars = smem_u32(base + C::kOffBars); off_misc = C::kOffMisc;
    }
    __device__ __forceinline__ uint32_t bar(int i) const { return bars + 8u * (uint32_t)i; }
    __device__ __forceinline__ uint8_t* b_ring() const { return base; }
    __device__ __forceinline__ uint8_t* s_slot(int s) const { return base + off_s + s * kSSlot; }
    __device__ __forceinline__ float* bias() const { return reinterpret_cast<float*>(base + off_bias); }
    __device__ __forceinline__ uint32_t* tmem_base() const { return reinterpret_cast<uint32_t*>(base + off_misc); }
    __device__ __forceinline__ volatile uint32_t* abort_flag() const {
        return reinterpret_cast<volatile uint32_t*>(base + off_misc + 4);
    }
};

// Hooks of a profiling build: a header given with -include may define them to sum clock64
// deltas per phase; in the library they expand to nothing.
#ifndef CFX_MARK
#define CFX_MARK_INIT(role)
#define CFX_MARK(bucket)
#define CFX_MARK_FLUSH()
#endif

// every role runs in its own function: a failed (timed-out) wait returns to the common exit
// Worker warps poll with try_wait (suspends while not ready).
// Measured alternatives, all slower on B200: one polling lane per worker warp plus a shuffle
// (+25 % kernel time), a test_wait probe in front of the loop (+6 %).
#define CFX_WAITW(barid, parity, code) \
    if (!mbar_wait_warp(sm.bar(barid), (parity), sm.abort_flag(), (code))) return
// the copy-issuing threads (one lane: loads, stores) and warp (weights): no back-off between probes
#define CFX_WAIT_FAST(barid, parity, code) \
    if (!mbar_wait<false>(sm.bar(barid), (parity), sm.abort_flag(), (code))) return
#define CFX_WAITW_FAST(barid, parity, code) \
    if (!mbar_wait_warp<false>(sm.bar(barid), (parity), sm.abort_flag(), (code))) return
// The MMA warp polls with test_wait: it never suspends.
#define CFX_WAIT_LEADER(barid, parity, code) \
    if (!mbar_wait_warp<false, true>(sm.bar(barid), (parity), sm.abort_flag(), (code))) return

// Who converts which operand chunk (a weight block's 64 K columns).  Group 0 samples the previous tile's actions while the
// other three convert: chunk kc is group 1 + kc % 3's.
constexpr int kExpGroups = kGroups - 1;

// ------------------------------------------------------------------ producer roles
// Weight stages, in the order of the MMAs: encoder (Cfg::kEncPer blocks), gate layers (layer, slice, half of a slice: all K
// blocks), heads; every tile replays the same sequence (the image stays L2 resident).
// In a CTA pair every CTA stages its own half of the rows of each
// block with a tensor copy whose completion is counted on the even
// CTA's "full" barrier, where the MMA warp waits; one CTA per tile uses plain bulk copies.
template <bool PAIR, int GAME, int HID>
__device__ __forceinline__ void role_weight_loads(const Smem& sm, const Params& P, uint32_t rank, uint32_t bar0_cta0) {
    using C = Cfg<PAIR, GAME, HID>;
    CFX_DIMS(HID);
    constexpr int kEncBlockBytes = Hd<HID>::kEncBlockBytes;
    const int enc_gate = C::kEncStages + P.L * C::kLayerStages;
    // The warp walks the launch-wide stage sequence and an elected lane issues: the slots come free in the order they were
    // filled.  A stage must not take longer here than its MMAs (520 to 790 cycles): with one lane walking alone it took
    // 750.  The next slot is probed before the copy into this one is issued.
    int tile = P.tile_begin + blockIdx.x, s = 0;
    int slot = 0;
    uint32_t par = 1;   // parity of the "empty" phase to wait for: the first pass finds every slot free
    CFX_MARK_INIT(3);
    CFX_PROBE(cfx_p_w, sm.bar(B_EMPTY + slot), par);
    for (; tile < P.num_tiles_loop;) {
        int region, row, blk;   // rows [row, ...) of blocks blk, blk + 1, ...
        uint32_t bytes;
        if (s < C::kEncStages) {
            region = 0; row = 0; blk = s * C::kEncPer;
            bytes = C::kCut ? min(C::kBSlot, Gm<GAME>::kEncBlocks * kEncBlockBytes - s * C::kBSlot) : C::kEncPer * kEncBlockBytes;
        } else if (s < enc_gate) {
            const int g = s - C::kEncStages;
            constexpr int kParts = kKBlocks / C::kGateKb;   // stages of half a slice
            region = 1; row = kHalfRows * (g / kParts & 1); blk = g / (2 * kParts) * kKBlocks + g % kParts * C::kGateKb;
            bytes = C::kGateKb * kHalfRows * 128;
        } else {
            region = 2; row = 0; blk = (int)rank; bytes = head_bytes<GAME, HID>(PAIR);
        }
        uint32_t ready;
        CFX_PROBE_READ_ALL(cfx_p_w, ready);
        if (ready == 0) CFX_WAITW_FAST(B_EMPTY + slot, par, W_B_EMPTY);
        const int slot1 = slot + 1 == C::kNB ? 0 : slot + 1;
        const uint32_t par1 = slot1 == 0 ? par ^ 1u : par;
        CFX_PROBE(cfx_p_w, sm.bar(B_EMPTY + slot1), par1);
        __syncwarp();
        CFX_MARK(1);
        const uint32_t dst = smem_u32(sm.b_ring() + slot * C::kBSlot), full = sm.bar(B_FULL + slot);
        if (PAIR) {
            // Each CTA copies its half of the rows into its own shared memory; both copies are
            // counted on the EVEN CTA's "full" barrier (where the MMA warp waits), which
            // expects the bytes of the whole stage.  The odd CTA needs no barrier of its own
            // and no forwarding hop.
            const int y = region == 0 ? C::kEncRows * (int)rank : (region == 1 ? row + C::kGateRows * (int)rank : 0);
            if (elect_one()) {
                if (rank == 0) mbar_arrive_expect_tx(full, bytes);
                tensor_g2s_3d_pair(dst, &P.w_map[region], 0, y, blk, bar0_cta0 + 8u * (uint32_t)(B_FULL + slot));
            }
        } else if (elect_one()) {
            mbar_arrive_expect_tx(full, bytes);
            const uint8_t* gates = P.image + enc_bytes<GAME, HID>();
            if (region == 0) {
                bulk_g2s(dst, P.image + (C::kCut ? (size_t)s * C::kBSlot : (size_t)blk * kEncBlockBytes), bytes, full);
            } else if (region == 1) {
#pragma unroll
                for (int b = 0; b < C::kGateKb; b++)
                    bulk_g2s(dst + b * kHalfRows * 128, gates + (size_t)(blk + b) * kGateBlockBytes + row * 128, kHalfRows * 128, full);
            } else {
                bulk_g2s(dst, gates + (size_t)P.L * kSlices * kKBlocks * kGateBlockBytes, bytes, full);
            }
        }
        CFX_MARK(2);
        if (++s > enc_gate) { s = 0; tile += gridDim.x; }
        slot = slot1; par = par1;
    }
    CFX_MARK_FLUSH();
}

// Records and state boxes.  Records: rows are contiguous in memory, sixteen are a copy (they were boxes of 128 rows x 80
// bytes a chunk, 64 copies a tile that took 850 cycles a chunk to issue).  State box: layer l, tile rows, 32 units -> one 16 KB
// box, 128-byte swizzled; box b of a tile (b counts through the layers) uses slot b % 8, so a layer's boxes come in while the
// layer before runs.  The workers replace a
// box's contents with the new state in place; it is then written back (rows beyond n are clipped by the tensor map).
//
// Two threads in two warps, each a plain sequence of waits and copies.  (Several
// lanes of one warp, one per ring slot, each in its own loop, ran at a fraction of that speed:
// a lane whose barrier had completed took 600-700 cycles to get from one statement to the
// next while the warp served the other lanes.)
//   load thread:  per tile, the records, then the state boxes, each when what was in its slots before is done with;
//   store thread: the state box stores; it reports a box that has been read out of its slot (S_FREE).
// Full game: the records of a CTA's first tile are loaded ahead of this by a lane a copy (see the kernel; the classic game's are one copy, and so 0.2 % slower).
// Copy i of a tile's records.  Rows [32 q, 32 q + 32) are a quadrant's (n is a multiple of 32): all of them are there or none, and then what lies
// in the slot is converted and multiplied like records, and the results of those rows are dropped.
template <bool PAIR, int GAME, int HID>
__device__ __forceinline__ void load_records(const Smem& sm, const Params& P, int tile, int i) {
    using C = Cfg<PAIR, GAME, HID>;
    const int r = i * C::kRecRows, row0 = tile * kTile + r, rows = min(C::kRecRows, P.n - row0);
    const uint32_t full = sm.bar(REC_FULL + r / 32);
    if (rows > 0) {
        mbar_arrive_expect_tx(full, (uint32_t)rows * C::kRecBytes);
        bulk_g2s(smem_u32(sm.s_slot(0)) + C::rec_offset(r), P.records + (size_t)row0 * C::kRecBytes, (uint32_t)rows * C::kRecBytes, full);
    } else {
        mbar_arrive(full);
    }
}

template <bool PAIR, int GAME, int HID, bool REC16>
__device__ __forceinline__ void role_loads(const Smem& sm, const Params& P) {
    using C = Cfg<PAIR, GAME, HID>;
    CFX_DIMS(HID);
    const int boxes = P.L * kStateItems;
    uint32_t it = 0;
    uint32_t fpar = 0;      // slots: parity of the "free" phase to wait for
    auto prefetch_records = [&](int tile, int i) {
        const int row0 = tile * kTile + 16 * i;
        if (tile < P.num_tiles && row0 < P.n) bulk_prefetch_l2(P.records + (size_t)row0 * C::kRecBytes, 16 * C::kRecBytes);
    };
    CFX_MARK_INIT(4);
    for (int tile = P.tile_begin + blockIdx.x; tile < P.num_tiles_loop; tile += gridDim.x, it++) {
        for (int u = 0; u < C::kRecSlots && (it > 0 || GAME != CFX_GAME_FULL); u++) {   // (full game, first tile: see the kernel)
            if (it > 0) {
                if (u >= boxes) {   // no state boxes here
                    if ((u & 1) == 0) CFX_WAIT_FAST(REC_FREE + u / 2, (it - 1) & 1, W_REC_FREE);
                } else {
                    CFX_WAIT_FAST(S_FREE + u, (fpar >> u) & 1u, W_S_FREE);
                    fpar ^= 1u << u;
                }
            }
            if (GAME == CFX_GAME_FULL) load_records<PAIR, GAME, HID>(sm, P, tile, u);
            else if (u == C::kRecSlots - 1) load_records<PAIR, GAME, HID>(sm, P, tile, 0);
            CFX_MARK(20 + u);
        }
        for (int b = 0; b < boxes; b++) {
            const int slot = b % kNS, l = b / kStateItems, j = b % kStateItems;
            if (GAME == CFX_GAME_FULL && b == C::kEarlyBoxes && (REC16 || P.r_state == nullptr)) CFX_WAIT_FAST(ACC_FULL, it & 1, W_ACC_FULL);
            if (b < C::kRecSlots) {
                if ((b & 1) == 0) CFX_WAIT_FAST(REC_FREE + b / 2, it & 1, W_REC_FREE);
            } else if (b >= kNS || it > 0) {
                CFX_WAIT_FAST(S_FREE + slot, (fpar >> slot) & 1u, W_S_FREE);
                fpar ^= 1u << slot;
            }
            CFX_MARK(1);
            mbar_arrive_expect_tx(sm.bar(S_FULL + slot), kSSlot);
            tensor_g2s_2d(smem_u32(sm.s_slot(slot)), &P.state_map[l], j * kHalfUnits, tile * kTile, sm.bar(S_FULL + slot));
            // What the next tile waits for last: where its boxes are whole rounds of the slots, the records of the last four.  (With 4
            // or 12 boxes, hidden 128 with one or three layers, the last four boxes are in slots 0 to 3, and those records wait the longest.
            // The classic game's are in the slots that come free first: without a prefetch as fast, 1,048,576 envs h256x3 2,216
            // and 2,231 us against 2,222 and 2,227.)
            if (GAME == CFX_GAME_FULL && b + kNS / 2 >= boxes) prefetch_records(tile + (int)gridDim.x, kNS + b - boxes);
            CFX_MARK(2);
        }
    }
    CFX_MARK_FLUSH();
}

template <bool PAIR, int GAME, int HID>
__device__ __forceinline__ void role_stores(const Smem& sm, const Params& P) {
    CFX_DIMS(HID);
    const int boxes = P.L * kStateItems;
    uint32_t spar = 0;                     // slots: parity of the "new state ready" phase
    CFX_MARK_INIT(5);
    for (int tile = P.tile_begin + blockIdx.x; tile < P.num_tiles_loop; tile += gridDim.x) {
        for (int b = 0; b < boxes; b++) {
            const int slot = b % kNS;
            CFX_WAIT_FAST(ST_READY + slot, (spar >> slot) & 1u, W_ST_READY);
            spar ^= 1u << slot;
            CFX_MARK(3);
            tensor_s2g_2d(&P.state_map[b / kStateItems], smem_u32(sm.s_slot(slot)), b % kStateItems * kHalfUnits, tile * kTile);
            bulk_commit_group();
            bulk_wait_group_read<0>();
            mbar_arrive(sm.bar(S_FREE + slot));
            CFX_MARK(4);
        }
    }
    bulk_wait_group<0>();
    CFX_MARK_FLUSH();
}

// ------------------------------------------------------------------ MMA role
// The whole warp walks through the steps, so that the compiler keeps descriptors and ring positions in uniform
// registers, and an elected lane issues every MMA of the CTA (262,144 envs h256x2 421 -> 412 us against one lane walking
// alone, 131,104 h128x2 bf16 123.1 -> 119.8, 65,536 h256x3 150.3 -> 148.5, classic 1,048,576 2,284 -> 2,236).  With every ring
// position a compile-time constant, the encoder and the four slices unrolled, the code is no faster and larger (417,
// 120.1, 148.8, 2,224).
// The tensor pipe queues four to five MMAs (a block of eight with N = 96 hides 150 cycles between blocks, with N = 192 500),
// so the issuer runs ahead of it as long as its own loop is short: descriptors are one add away from
// a per-slot base and the sixteen MMAs of half a slice are one straight run (33 cycles an MMA; rebuilding descriptors per MMA
// measured ~150).
#define MMA_TS(...)                                  \
    do {                                             \
        if (PAIR) mma_f16_ts_pair(__VA_ARGS__);      \
        else mma_f16_ts(__VA_ARGS__);                \
    } while (0)
// commits: in a pair they arrive on the barrier of BOTH CTAs
#define MMA_COMMIT(bar)                  \
    do {                                 \
        if (PAIR) mma_commit_pair(bar);  \
        else mma_commit(bar);            \
    } while (0)
template <typename T16, bool PAIR, int GAME, int HID>
__device__ __forceinline__ void role_mma(const Smem& sm, const Params& P, uint32_t tmem) {
    using C = Cfg<PAIR, GAME, HID>;
    CFX_DIMS(HID);
    constexpr int kEncBlocks = Gm<GAME>::kEncBlocks;
    constexpr int kNB = C::kNB, kBSlot = C::kBSlot;
    constexpr uint32_t fmt = Op16<T16>::kFmt;
    constexpr uint32_t idesc_enc = make_idesc(fmt, C::kM, kH);
    constexpr uint32_t idesc_gate = make_idesc(fmt, C::kM, kHalfRows);
    constexpr uint32_t idesc_head = make_idesc(fmt, C::kM, C::kHeadRows);
    // descriptor steps (16-byte units) between the blocks of a stage
    constexpr uint32_t kEncBlkStep = (C::kEncRows * 128) >> 4, kGateBlkStep = (C::kGateRows * 128) >> 4;
    const uint64_t bdesc0 = smem_desc_sw128(smem_u32(sm.b_ring()));
    uint32_t acnt = 0, akb_use = 0, gcnt = 0, tcnt = 0;
    // position in the weight ring of the stage being consumed: slot and phase parity, advanced
    // incrementally (a division per stage of this warp would sit on the critical path)
    int bslot = 0;
    uint32_t bpar = 0;
    auto b_advance = [&]() {
        if (++bslot == kNB) { bslot = 0; bpar ^= 1u; }
    };
    // The "full" barriers of the NEXT stage are probed before the current stage's MMAs are
    // issued, so that the probe's shared-memory round trip (~150 cycles on this thread) runs
    // under the MMA issue; only a failed probe falls into the bounded wait.  Probing one stage
    // early is sound: the previous use of that slot has already been consumed by this thread,
    // so its barrier is at most one phase behind.
    // The probes are deferred ones (CFX_PROBE): their result is read a stage later.
    auto probe_b_next = [&]() {
        const bool wrap = bslot + 1 == kNB;
        CFX_PROBE(cfx_p_b, sm.bar(B_FULL + (wrap ? 0 : bslot + 1)), wrap ? bpar ^ 1u : bpar);
    };
    auto probe_a = [&](uint32_t cnt) {
        CFX_PROBE(cfx_p_a, sm.bar(AEXP_FULL + (int)(cnt % kAexpSlots)), (cnt / kAexpSlots) & 1);
    };
    // the four K steps of K block kb against its rows of the stage at bd0, for half h of a slice
    auto gate_mmas = [&](int h, int kb, uint32_t a_cur, uint64_t bd0) {
#pragma unroll
        for (int ks = 0; ks < 4; ks++)
            MMA_TS(tmem + kColG + h * kHalfRows, a_cur + kb * 32 + ks * 8, bd0 + (uint64_t)(kb % C::kGateKb * kGateBlkStep + 2 * ks), idesc_gate,
                   (kb | ks) != 0 ? 1u : 0u);
    };
#define CFX_WAIT_PROBED(name, barid, parity, code)                                                  \
    {                                                                                               \
        uint32_t ready_;                                                                            \
        CFX_PROBE_READ_ALL(name, ready_);                                                               \
        if (ready_ == 0) CFX_WAIT_LEADER(barid, parity, code);             \
    }
    CFX_PROBE(cfx_p_ge, sm.bar(G_EMPTY), 1);
    CFX_MARK_INIT(0);
    for (int tile = P.tile_begin + blockIdx.x; tile < P.num_tiles_loop; tile += gridDim.x, tcnt++) {
        CFX_MARK(0);
        // the encoder accumulator overlaps the head accumulator of the previous tile:
        // wait until the sampler threads have read it
        CFX_WAIT_LEADER(H_EMPTY, (tcnt & 1) ^ 1, W_H_EMPTY);
        probe_a(acnt);
        CFX_PROBE(cfx_p_b, sm.bar(B_FULL + bslot), bpar);
        // ---- encoder: N = kH units; a block of 64 K columns is one operand chunk
        // the K steps of a block against n units of it from `unit` on, at bd
        auto enc_mmas = [&](uint32_t a_col, uint64_t bd, bool first, bool last, int unit, int n) {
            const uint32_t d = tmem + kColAcc + unit, idesc = n == kH ? idesc_enc : make_idesc(fmt, C::kM, n);
            // the last block has 25 features (full game: two K steps) or one (classic: one K step)
            MMA_TS(d, a_col, bd, idesc, first ? 0u : 1u);
            if (GAME == CFX_GAME_FULL || !last) MMA_TS(d, a_col + 8, bd + 2, idesc, 1);
            if (!last) {
                MMA_TS(d, a_col + 16, bd + 4, idesc, 1);
                MMA_TS(d, a_col + 24, bd + 6, idesc, 1);
            }
        };
        if constexpr (C::kCut) {   // a block is multiplied in two parts, from the stage that its first units are in and from the next one
            int slot = 0;
            for (int kc0 = 0; kc0 < kEncBlocks; kc0 += 3) {
#pragma unroll
                for (int q = 0; q < 3; q++, acnt++) {   // the first q kCutUnit rows of the stage were the block before's
                    const int kc = kc0 + q, as = acnt % kAexpSlots, n0 = C::kCutRows - C::kCutUnit * q;
                    if (kc >= kEncBlocks) break;
                    const bool last = kc == kEncBlocks - 1;
                    if (q == 0) {
                        slot = bslot;
                        CFX_WAIT_PROBED(cfx_p_b, B_FULL + slot, bpar, W_B_FULL);
                        probe_b_next();
                        b_advance();
                    }
                    CFX_WAIT_PROBED(cfx_p_a, AEXP_FULL + as, (acnt / kAexpSlots) & 1, W_AEXP_FULL);
                    if (!last) probe_a(acnt + 1);
                    tc_fence_after_sync();
                    __syncwarp();
                    const uint32_t a_col = tmem + kColAexp + as * 32;
                    if (elect_one()) {
                        enc_mmas(a_col, bdesc0 + (uint64_t)(slot * (kBSlot >> 4) + ((q * C::kCutUnit * 128) >> 4)), kc == 0, last, 0, n0);
                        MMA_COMMIT(sm.bar(B_EMPTY + slot));
                    }
                    slot = bslot;
                    CFX_WAIT_PROBED(cfx_p_b, B_FULL + slot, bpar, W_B_FULL);
                    probe_b_next();
                    b_advance();
                    tc_fence_after_sync();
                    __syncwarp();
                    if (elect_one()) {
                        enc_mmas(a_col, bdesc0 + (uint64_t)(slot * (kBSlot >> 4)), kc == 0, last, n0, kH - n0);
                        MMA_COMMIT(sm.bar(AEXP_EMPTY + as));
                        if (q == 2 || last) MMA_COMMIT(sm.bar(B_EMPTY + slot));
                        if (last) MMA_COMMIT(sm.bar(ACC_FULL));
                    }
                }
            }
        } else for (int kc = 0; kc < kEncBlocks; kc += C::kEncPer) {
            const int slot = bslot;
            CFX_WAIT_PROBED(cfx_p_b, B_FULL + slot, bpar, W_B_FULL);
            CFX_MARK(3);
            probe_b_next();
            b_advance();
#pragma unroll
            for (int c2 = 0; c2 < C::kEncPer; c2++, acnt++) {
                const int as = acnt % kAexpSlots;
                const bool last = c2 == C::kEncPer - 1 && kc + C::kEncPer == kEncBlocks;
                CFX_WAIT_PROBED(cfx_p_a, AEXP_FULL + as, (acnt / kAexpSlots) & 1, W_AEXP_FULL);
                CFX_MARK(2);
                if (!last) probe_a(acnt + 1);
                tc_fence_after_sync();
                __syncwarp();
                const uint32_t a_col = tmem + kColAexp + as * 32;
                const uint64_t bd = bdesc0 + (uint64_t)(slot * (kBSlot >> 4) + c2 * kEncBlkStep);
                if (elect_one()) {
                    enc_mmas(a_col, bd, c2 == 0 && kc == 0, last, 0, kH);
                    MMA_COMMIT(sm.bar(AEXP_EMPTY + as));
                    if (c2 == C::kEncPer - 1) MMA_COMMIT(sm.bar(B_EMPTY + slot));
                    if (last) MMA_COMMIT(sm.bar(ACC_FULL));
                }
                CFX_MARK(4);
            }
        }

        // ---- MinGRU layers: slices of 64 units in two halves, each with an accumulator of its own (N = 96: zh|zg|zp of 32
        // units), so that one half is multiplied while the workers take the other one's
        for (int l = 0; l < P.L; l++, akb_use++) {
            const uint32_t a_cur = tmem + ((l & 1) ? kColA1 : kColA0);
            for (int j = 0; j < kSlices; j++, gcnt++) {
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    CFX_WAIT_PROBED(cfx_p_ge, G_EMPTY + h, (gcnt & 1) ^ 1, W_G_EMPTY);
                    CFX_MARK(5);
                    // The gate accumulators overlap the encoder accumulator: the first gate MMA of a
                    // tile waits until every worker warp has moved its part of it to registers.
                    // (An early version waited only for the K block it multiplied while a warpgroup
                    // was still reading the accumulator: about one launch in a hundred changed 32
                    // rows of one tile.)
                    if (h == 0 && l == 0 && j == 0) {
                        CFX_WAIT_LEADER(ACC_READ, tcnt & 1, W_ACC_READ);
                        CFX_MARK(9);
                    }
#pragma unroll
                    for (int kp = 0; kp < kKBlocks; kp += C::kGateKb) {
                        const int slot = bslot;
                        CFX_WAIT_PROBED(cfx_p_b, B_FULL + slot, bpar, W_B_FULL);
                        CFX_MARK(6);
                        probe_b_next();
                        b_advance();
                        const uint64_t bd0 = bdesc0 + (uint64_t)(slot * (kBSlot >> 4));
                        if (h == 0 && j == 0) {   // the layer's input arrives K block by K block (slice kb of the previous layer)
                            for (int kb = kp; kb < kp + C::kGateKb; kb++) {
                                CFX_WAIT_LEADER(A_KB + kb, akb_use & 1, W_A_KB);
                                CFX_MARK(9);
                                tc_fence_after_sync();
                                __syncwarp();
                                if (elect_one()) gate_mmas(h, kb, a_cur, bd0);
                            }
                        } else {
                            tc_fence_after_sync();
                            __syncwarp();
                            if (elect_one()) {
#pragma unroll
                                for (int kb = kp; kb < kp + C::kGateKb; kb++) gate_mmas(h, kb, a_cur, bd0);
                            }
                        }
                        __syncwarp();
                        // (the other half's accumulator: handed back while this half is multiplied)
                        const bool ends = kp + C::kGateKb == kKBlocks;
                        if (ends) CFX_PROBE(cfx_p_ge, sm.bar(G_EMPTY + (h ^ 1)), ((gcnt + h) & 1) ^ 1);
                        if (elect_one()) {
                            if (ends) MMA_COMMIT(sm.bar(G_FULL + h));
                            MMA_COMMIT(sm.bar(B_EMPTY + slot));
                        }
                        CFX_MARK(7);
                    }
                }
            }
        }
        // ---- heads: N = 48 (64 in a pair), one stage with all K blocks
        {
            const uint32_t a_cur = tmem + ((P.L & 1) ? kColA1 : kColA0);
            const int slot = bslot;
            CFX_WAIT_PROBED(cfx_p_b, B_FULL + slot, bpar, W_B_FULL);
            b_advance();
            const uint64_t bd = bdesc0 + (uint64_t)(slot * (kBSlot >> 4));
            // K block kb of the last layer's output is complete when slice kb's cells are done
#pragma unroll
            for (int kb = 0; kb < kKBlocks; kb++) {
                CFX_WAIT_LEADER(A_KB + kb, akb_use & 1, W_A_KB);
                tc_fence_after_sync();
                __syncwarp();
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < 4; ks++)
                        MMA_TS(tmem + kColHead, a_cur + kb * 32 + ks * 8,
                               bd + (uint64_t)((kb * C::kHeadKbBytes + ks * 32) >> 4), idesc_head,
                               (kb | ks) != 0 ? 1u : 0u);
                    if (kb == kKBlocks - 1) {
                        MMA_COMMIT(sm.bar(B_EMPTY + slot));
                        MMA_COMMIT(sm.bar(H_FULL));
                    }
                }
            }
            akb_use++;
            CFX_MARK(8);
        }
    }
    CFX_MARK_FLUSH();
}

// ------------------------------------------------------------------ worker role
// Sixteen warps, four per TMEM lane quarter (groups wg 0 to 3); thread (quarter, lane) owns env row
// quarter*32 + lane of the tile in every phase.
template <typename T16, bool PAIR, int GAME, int HID, bool REC16>
__device__ __forceinline__ void role_worker(const Smem& sm, const Params& P, uint32_t tmem,
                                            int warp, int lane, uint32_t bar0_cta0) {
    using Op = Op16<T16>;
    using C = Cfg<PAIR, GAME, HID>;
    CFX_DIMS(HID);
    constexpr int kEncBlocks = Gm<GAME>::kEncBlocks, kA = Gm<GAME>::kA;
    constexpr int kHeadCols = (kA + 1 + 15) / 16 * 16;   // head accumulator columns that are read
    // barriers the MMA warp waits on live in the even CTA of a pair
    auto arrive_mma = [&](int barid) {
        if (PAIR) mbar_arrive_cluster(bar0_cta0 + 8u * (uint32_t)barid);
        else mbar_arrive(sm.bar(barid));
    };
    const int wg = (warp - kWorkerWarp0) >> 2;
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const int half = wg >> 1;   // of a slice
    const uint8_t* rec = sm.s_slot(0) + C::rec_offset(row);
    const float* bias = sm.bias();
    uint32_t tcnt = 0, gcnt = 0, it = 0;
    uint32_t spar = 0;   // phase parity of every state slot, one bit per slot
    // (classic game, whose kernel has the registers; read for every tile: 1,048,576 envs h256x3 2,207 and 2,209)
    const unsigned long long step0 = GAME == CFX_GAME_CLASSIC && P.uniforms == nullptr ? *P.step_ctr : 0ull;
    CFX_MARK_INIT(1);
    for (int tile = P.tile_begin + blockIdx.x; tile < P.num_tiles_loop; tile += gridDim.x, it++, tcnt++) {
        CFX_MARK(0);
        const int env = tile * kTile + row;
        const bool valid = env < P.n;
        float terminal = 0.0f;
        if (valid && P.prev_terminals != nullptr) terminal = P.prev_terminals[env];

        // ---- expand: record bytes -> 16-bit operand rows in the TMEM chunk ring.
        // A warp writes all columns of its rows.  The operand slot's barrier is probed one chunk ahead, so that the
        // probe's shared-memory round trip (~200 cycles, also when the barrier is already
        // complete) runs under the previous chunk's conversion; only a failed probe falls into
        // the wait loop.
        float u = 0.0f;
        if (wg > 0) {
            uint32_t acnt = it * kEncBlocks + wg - 1;
            CFX_PROBE(cfx_p_ae, sm.bar(AEXP_EMPTY + (int)(acnt % kAexpSlots)), ((acnt / kAexpSlots) & 1) ^ 1);
            CFX_WAITW(REC_FULL + quarter * C::kRecSlots / 8, it & 1, W_REC_FULL);
            CFX_MARK(3);
            for (int kc = wg - 1; kc < kEncBlocks; kc += kExpGroups, acnt += kExpGroups) {
                const int as = acnt % kAexpSlots;
                uint32_t ae_ok;
                CFX_PROBE_READ_ALL(cfx_p_ae, ae_ok);
                if (ae_ok == 0) CFX_WAITW(AEXP_EMPTY + as, ((acnt / kAexpSlots) & 1) ^ 1, W_AEXP_EMPTY);
                CFX_MARK(2);
                tc_fence_after_sync();
                const bool more = kc + kExpGroups < kEncBlocks;
                if (more) {
                    const uint32_t acnt1 = acnt + kExpGroups;
                    CFX_PROBE(cfx_p_ae, sm.bar(AEXP_EMPTY + (int)(acnt1 % kAexpSlots)), ((acnt1 / kAexpSlots) & 1) ^ 1);
                }
                uint32_t lo[16], hi[16];
                {
                    uint32_t regs[32];
                    if constexpr (GAME == CFX_GAME_CLASSIC) expand_classic<Op>(rec, kc, regs);
                    else expand_block<Op>(rec, kc, regs);
#pragma unroll
                    for (int q = 0; q < 16; q++) { lo[q] = regs[q]; hi[q] = regs[16 + q]; }
                }
                if (!more) {   // this warp has read its last record byte of the tile
                    __syncwarp();
                    if (lane == 0) mbar_arrive(sm.bar(REC_FREE + quarter * C::kRecSlots / 8));
                }
                tmem_st16(tmem + lane_base + kColAexp + as * 32, lo);
                tmem_st16(tmem + lane_base + kColAexp + as * 32 + 16, hi);
                tmem_wait_st();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) arrive_mma(AEXP_FULL + as);
                CFX_MARK(4);
            }
        } else if (valid) {   // the uniform of this env is drawn while the others convert
            // (The step counter is constant for the launch: it is raised when every block is done.  Full game: read once and kept in registers
            // through the tiles, and so, us: h128x2 24,064 envs 27.9 and 27.1, 57,600 53.5 and 52.7; h256x2 20,000 41.5 and 41.3.)
            u = P.uniforms != nullptr ? P.uniforms[env] : philox_uniform(P.seed, P.env_offset + (uint64_t)env, GAME == CFX_GAME_CLASSIC ? step0 : *P.step_ctr);
        }

        // ---- encoder epilogue: accumulator + bias -> layer-0 input A0.  Like in the gate
        // layers, group wg handles units [64 kb + 16 wg, 64 kb + 16 wg + 16) of K block kb.
        // The whole accumulator goes to registers first and is handed back at once (ACC_READ):
        // the gate accumulator overlaps it, and the first slice's MMAs then start on K block 0
        // while the later blocks are still being converted.
        CFX_WAITW(ACC_FULL, tcnt & 1, W_ACC_FULL);
        CFX_MARK(5);
        tc_fence_after_sync();
        {
            uint32_t acc[kKBlocks][kWarpUnits];
#pragma unroll
            for (int kb = 0; kb < kKBlocks; kb++)
                tmem_ld16(tmem + lane_base + kColAcc + kSliceUnits * kb + kWarpUnits * wg, acc[kb]);
            tmem_wait_ld();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) arrive_mma(ACC_READ);
#pragma unroll
            for (int kb = 0; kb < kKBlocks; kb++) {
                uint32_t pk[kWarpUnits / 2];
                const float* bb = bias + kSliceUnits * kb + kWarpUnits * wg;
#pragma unroll
                for (int q = 0; q < kWarpUnits / 2; q++)
                    pk[q] = Op::pack(__uint_as_float(acc[kb][2 * q]) + bb[2 * q],
                                     __uint_as_float(acc[kb][2 * q + 1]) + bb[2 * q + 1]);
                tmem_st8(tmem + lane_base + kColA0 + (kSliceUnits / 2) * kb + (kWarpUnits / 2) * wg, pk);
                tmem_wait_st();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) arrive_mma(A_KB + kb);
            }
        }
        CFX_MARK(1);

        // ---- MinGRU layers: groups 0 and 1 have the first half of every 64-unit slice, 2 and 3 the second; wg handles units
        // [64 j + 16 wg, 64 j + 16 wg + 16), half of state box 2 j + wg / 2 of the layer
        // Here too the next barrier is probed while other work runs: the state box while the
        // accumulator is read, the next accumulator (or the heads) while the cell's last stores
        // drain.
        CFX_PROBE_CLEAR(cfx_p_g);
        asm volatile("" : "+f"(terminal));   // (not looked at before: the tile's start would wait for it)
        const bool zero_state = terminal != 0.0f;
        for (int l = 0; l < P.L; l++) {
            const uint32_t a_cur = tmem + lane_base + ((l & 1) ? kColA1 : kColA0);
            const uint32_t a_next = tmem + lane_base + ((l & 1) ? kColA0 : kColA1);
            for (int j = 0; j < kSlices; j++, gcnt++) {
                const int slot = (l * kStateItems + 2 * j + half) % kNS;
                const uint32_t sp_par = (spar >> slot) & 1u;
                spar ^= 1u << slot;
                // under the slice's MMAs (of a warp's rows all or none are valid).  The ballot of the flags stands here and not at
                // the tile's start, where it would wait for them: 65,536 envs h256x3 145.7 -> 142.8 us, one set of buffers
                if (!REC16 && P.r_state != nullptr && valid) {
                    CFX_WAITW(S_FULL + slot, sp_par, W_S_FULL);
                    write_r_state<4, kH>(P, sm.s_slot(slot) + quarter * 4096, 4 * (wg & 1),
                                         ((size_t)l * P.n + tile * kTile + quarter * 32) * kH + kSliceUnits * j + kWarpUnits * wg,
                                         __ballot_sync(0xffffffffu, zero_state), lane);
                }
                {
                    uint32_t g_ok;
                    CFX_PROBE_READ_ALL(cfx_p_g, g_ok);
                    if (g_ok == 0) CFX_WAITW(G_FULL + half, gcnt & 1, W_G_FULL);
                }
                CFX_MARK(6);
                tc_fence_after_sync();
                CFX_PROBE(cfx_p_s, sm.bar(S_FULL + slot), sp_par);
                const uint32_t gcol = tmem + lane_base + kColG + gate_row(0, kWarpUnits * wg);
                uint8_t* rbase = sm.s_slot(slot) + (row >> 3) * 1024 + (row & 7) * 128;
                const int xr = row & 7;
                // this thread's 48 gate columns and 16 layer inputs go to registers at once, so
                // the accumulator is handed back to the MMA warp right away
                uint32_t zh[kWarpUnits], zg[kWarpUnits], zp[kWarpUnits], xin[kWarpUnits / 2];
                tmem_ld16(gcol, zh);
                tmem_ld16(gcol + kWarpUnits, zg);
                tmem_ld16(gcol + 2 * kWarpUnits, zp);
                tmem_ld8(a_cur + (kSliceUnits / 2) * j + (kWarpUnits / 2) * wg, xin);
                tmem_wait_ld();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) arrive_mma(G_EMPTY + half);
                CFX_MARK(7);
                {
                    uint32_t s_ok;
                    CFX_PROBE_READ_ALL(cfx_p_s, s_ok);
                    if (s_ok == 0) CFX_WAITW(S_FULL + slot, sp_par, W_S_FULL);
                }
                CFX_MARK(8);
                uint32_t hn[kWarpUnits / 2];
                float rs[kWarpUnits / 2];   // REC16: the state record of this thread's units, packed
                // REC16: the thread's state is read before its cells, since the record waits for all of it: with a bf16 record h128x2 18,944 envs
                // 18.31 -> 17.98 us, 57,600 59.4 -> 58.0, h256x2 16,416 29.1 -> 29.0. Without such a record the registers that this takes cost 1.5 to 3 %
                float4 own[REC16 ? kWarpUnits / 4 : 1];
                if (REC16) {
#pragma unroll
                    for (int q = 0; q < kWarpUnits / 4; q++) own[q] = *reinterpret_cast<const float4*>(rbase + (((4 * (wg & 1) + q) ^ xr) << 4));
                }
#pragma unroll
                for (int q = 0; q < kWarpUnits / 4; q++) {
                    const int u = 4 * q;  // first of four units
                    float4* sp = reinterpret_cast<float4*>(rbase + (((4 * (wg & 1) + q) ^ xr) << 4));
                    float4 st = REC16 ? own[REC16 ? q : 0] : *sp;
                    if (zero_state) st = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (REC16) {
                        rs[2 * q] = __uint_as_float(Op16<__nv_bfloat16>::pack(st.x, st.y));
                        rs[2 * q + 1] = __uint_as_float(Op16<__nv_bfloat16>::pack(st.z, st.w));
                        if (q == kWarpUnits / 4 - 1 && valid)
                            st_global_v8(reinterpret_cast<float*>(reinterpret_cast<__nv_bfloat16*>(P.r_state) + ((size_t)l * P.n + env) * kH + kSliceUnits * j + kWarpUnits * wg), rs);
                    }
                    const float2 x01 = Op::unpack(xin[u / 2]), x23 = Op::unpack(xin[u / 2 + 1]);
                    float4 out;
                    float h0, h1, h2, h3;
                    mingru_cell_pair(__uint_as_float(zh[u]), __uint_as_float(zh[u + 1]),
                                     __uint_as_float(zg[u]), __uint_as_float(zg[u + 1]),
                                     __uint_as_float(zp[u]), __uint_as_float(zp[u + 1]),
                                     st.x, st.y, x01.x, x01.y, out.x, out.y, h0, h1);
                    mingru_cell_pair(__uint_as_float(zh[u + 2]), __uint_as_float(zh[u + 3]),
                                     __uint_as_float(zg[u + 2]), __uint_as_float(zg[u + 3]),
                                     __uint_as_float(zp[u + 2]), __uint_as_float(zp[u + 3]),
                                     st.z, st.w, x23.x, x23.y, out.z, out.w, h2, h3);
                    *sp = out;
                    hn[2 * q] = Op::pack(h0, h1);
                    hn[2 * q + 1] = Op::pack(h2, h3);
                }
                tmem_st8(a_next + (kSliceUnits / 2) * j + (kWarpUnits / 2) * wg, hn);
                // the next accumulator: the heads after the last slice of the last layer
                if (l == P.L - 1 && j == kSlices - 1) CFX_PROBE(cfx_p_g, sm.bar(H_FULL), tcnt & 1);
                else CFX_PROBE(cfx_p_g, sm.bar(G_FULL + half), (gcnt + 1) & 1);
                tmem_wait_st();
                tc_fence_before_sync();
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    arrive_mma(A_KB + j);
                    mbar_arrive(sm.bar(ST_READY + slot));
                }
                CFX_MARK(9);
            }
        }

        // ---- heads + sampler (wg 0: one thread per env; the others only pass the barrier so
        // that their next-tile operand writes cannot overtake the last MMA)
        {
            uint32_t h_ok;
            CFX_PROBE_READ_ALL(cfx_p_g, h_ok);
            if (h_ok == 0) CFX_WAITW(H_FULL, tcnt & 1, W_H_FULL);
        }
        CFX_MARK(10);
        tc_fence_after_sync();
        if (wg == 0) {
            uint32_t hv[kHeadCols];
#pragma unroll
            for (int b = 0; b < kHeadCols / 16; b++) {
                uint32_t t[16];
                tmem_ld16(tmem + lane_base + kColHead + 16 * b, t);
#pragma unroll
                for (int q = 0; q < 16; q++) hv[16 * b + q] = t[q];
            }
            tmem_wait_ld();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) arrive_mma(H_EMPTY);
            if (valid) {
                write_outputs<GAME>(P, env, hv, bias + kH, u);
            }
            CFX_MARK(11);
        }
    }
    CFX_MARK_FLUSH();
}

// ------------------------------------------------------------------ kernel
// PAIR = false: one CTA per 128-env tile.  PAIR = true: launched as clusters of two CTAs; CTA r
// of a pair owns tile 2 c + r in every respect (records, state, expand, cell, sampler) except
// that the MMA warp of the even CTA issues one 256-row MMA for both tiles and every CTA
// stages only its half of the weight rows.
template <typename T16, bool PAIR, int GAME, int HID, bool REC16>
__global__ void __launch_bounds__(kThreads, 1)
k_policy_fused(const __grid_constant__ Params P) {
    using C = Cfg<PAIR, GAME, HID>;
    CFX_DIMS(HID);
    constexpr int kA = Gm<GAME>::kA;
    // predicates of the deferred probes: weight loads, MMA warp (gate accumulators, weights, operand chunks), workers (operand
    // slot, state box, next accumulator)
    CFX_PROBE_DECL(cfx_p_b);
    CFX_PROBE_DECL(cfx_p_a);
    CFX_PROBE_DECL(cfx_p_w);
    CFX_PROBE_DECL(cfx_p_ge);
    CFX_PROBE_DECL(cfx_p_ae);
    CFX_PROBE_DECL(cfx_p_s);
    CFX_PROBE_DECL(cfx_p_g);
    extern __shared__ uint8_t smem_raw[];
    Smem sm;
    sm.base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    sm.template layout<PAIR, GAME, HID>();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
    // arrivals per phase on the barriers the MMA warp waits on: both CTAs' workers in a pair
    const uint32_t both = (PAIR && rank == 0) ? 2u : 1u;

    if (tid == 0) {
        auto init = [&](int first, int count, uint32_t arrivals) {
            for (int i = 0; i < count; i++) mbar_init(sm.bar(first + i), arrivals);
        };
        init(B_FULL, C::kNB, 1);   // pair: the even CTA's barrier also counts the odd CTA's bytes
        init(B_EMPTY, C::kNB, 1);
        init(S_FULL, kNS, 1);
        init(S_FREE, kNS, 1);
        init(ST_READY, kNS, 8);            // two groups have a box
        init(REC_FULL, 4, 32 / C::kRecRows > 1 ? 32 / C::kRecRows : 1);   // copies of a quadrant (classic: one for all)
        init(REC_FREE, C::kRecSlots / 2, kExpGroups * 8 / C::kRecSlots);   // the warps that convert, after their last chunk
        init(AEXP_FULL, kAexpSlots, 4 * both);
        init(AEXP_EMPTY, kAexpSlots, 1);
        init(ACC_FULL, 1, 1);
        init(A_KB, kKBlocks, kWorkerWarps * both);
        init(G_FULL, 2, 1);
        init(G_EMPTY, 2, kWorkerWarps / 2 * both);
        init(H_FULL, 1, 1);
        init(H_EMPTY, 1, 4 * both);
        init(ACC_READ, 1, kWorkerWarps * both);
        *sm.abort_flag() = 0;
        fence_mbar_init();
    }
    if (warp == 1) {
        if (PAIR) {
            tmem_alloc_pair(smem_u32(sm.tmem_base()), 512);
            tmem_relinquish_pair();
        } else {
            tmem_alloc(smem_u32(sm.tmem_base()), 512);
            tmem_relinquish();
        }
    }
    if (warp == 3 && lane == 31) {
        for (int l = 0; l < P.L; l++) prefetch_tensormap(&P.state_map[l]);
    }
    // The next kernel may start its own set-up as soon as SMs come free.  The operand image and the biases are only
    // ever written by calls that wait for the device, so they may be read while the kernel in front in the stream
    // still runs; the roles that touch anything else wait for it.
    launch_next_kernel();
    for (int i = tid; i < kH + kHeadMax; i += kThreads) {
        float v = 0.0f;
        if (i < kH) v = P.params[P.off_b_enc + i];
        else if (i - kH < kA) v = P.params[P.off_b_a + (i - kH)];
        else if (i - kH == kA) v = P.params[P.off_b_v];
        sm.bias()[i] = v;
    }
    tc_fence_before_sync();
    // in a pair the peer's barriers must be initialised before anybody arrives on them
    if (PAIR) cluster_sync_all();
    else __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *sm.tmem_base();
    const uint32_t bar0_cta0 = PAIR ? map_to_cta(sm.bar(0), 0u) : 0u;

    if (warp < kWorkerWarp0) {
        if (warp == 0) {
            role_weight_loads<PAIR, GAME, HID>(sm, P, rank, bar0_cta0);
        } else if (warp == 1) {
            if (rank == 0) role_mma<T16, PAIR, GAME, HID>(sm, P, tmem);
        } else {
            // The first tile's records, a lane a copy: issued one behind the other they were 500 cycles apart.  us a step, h256x2 9,504 envs 24.3 -> 24.0,
            // 18,944 28.4 -> 27.9, h128x2 16,160 17.0 -> 16.6, 20,000 28.2 -> 27.5.
            const int first = P.tile_begin + (int)blockIdx.x;
            wait_for_previous_kernel();
            if constexpr (GAME == CFX_GAME_FULL) {
                if (warp == 2 && lane < C::kRecCopies && first < P.num_tiles_loop) load_records<PAIR, GAME, HID>(sm, P, first, lane);
                __syncwarp();
            }
            if (lane == 0) {
                if (warp == 2) role_loads<PAIR, GAME, HID, REC16>(sm, P);
                else role_stores<PAIR, GAME, HID>(sm, P);
            }
        }
    } else {
        // A CTA that has an SM to itself before the kernel in front has ended, because the CTA there had a tile less, asks for its first tile's records
        // to be brought into L2 meanwhile (not a read: what that kernel may still write to them is seen).  us a step without and with it: h256x2 20,000 envs
        // 41.7 and 40.8, 37,888 58.3 and 57.2, 65,536 104.8 and 102.4, 262,144 378.5 and 376.6; h128x2 28,416 28.9 and 28.0, 131,104 102.2 and 100.3.  A pass by
        // itself, with no kernel in front: h256x2 20,480 57.1 and 57.7, 37,888 60.9 and 61.0, 262,144 341.2 and 341.1; h128x2 131,104 109.9 and 109.8.  Where every
        // CTA has one tile they end together, and it is slower (18,944 28.2 and 28.6, h128x2 17.3 and 17.7).  The classic game's records are a seventh: no difference.
        if (GAME == CFX_GAME_FULL && P.num_tiles_loop - P.tile_begin > (int)gridDim.x) {
            const int row0 = (P.tile_begin + (int)blockIdx.x) * kTile, bytes = min(kTile, P.n - row0) * C::kRecBytes;
            const uint8_t* const p = P.records + (size_t)row0 * C::kRecBytes;
            for (int i = (tid - 32 * kWorkerWarp0) * 128; i < bytes; i += 32 * kWorkerWarps * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + i));
        }
        wait_for_previous_kernel();
        role_worker<T16, PAIR, GAME, HID, REC16>(sm, P, tmem, warp, lane, bar0_cta0);
    }

    // common exit: every role ends here, also after a timed-out wait.  In a pair neither CTA
    // may release its shared and tensor memory while the peer can still signal or read it.
    __syncwarp();
    tc_fence_before_sync();
    if (PAIR) cluster_sync_all();
    else __syncthreads();
    const uint32_t aborted = *sm.abort_flag();
    if (aborted != 0) {
        if (tid == 0) *reinterpret_cast<volatile uint32_t*>(P.status) = aborted | ((uint32_t)blockIdx.x << 8);
        // give copies that are still in flight time to land before shared memory is released
        for (int i = 0; i < 64; i++) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 1) {
        if (PAIR) tmem_dealloc_pair(tmem, 512);
        else tmem_dealloc(tmem, 512);
    }
    // every block read the counter (in its sampler threads) before it got here
    if (tid == 0 && P.bump_step) done_with_step(P.step_ctr, P.done_ctr, P.done_blocks);
}

// Self-test of the bounded wait: the first warp of a block waits with a limit of a few milliseconds, every other lane on a
// phase that is complete, the rest on a barrier on which nothing ever arrives.  All of its lanes give up together (kSelftestParted
// if some go on), and it reports through the same status word
// protocol as the forward kernels.  The second warp is at the first of the two meetings it has with the first one by then,
// and is let go; it alone has said that it is done with the step counter.  The kernel ends normally; the context stays
// usable.
constexpr uint32_t kSelftestCode = 0x7E, kSelftestParted = 0x7F;
__global__ void k_selftest_wait_timeout(uint32_t* status, uint32_t* done, unsigned long long limit_ns) {
    __shared__ uint64_t bar[2];
    __shared__ uint32_t abort_flag;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        mbar_init(smem_u32(&bar[0]), 1);
        mbar_init(smem_u32(&bar[1]), 1);
        fence_mbar_init();
        mbar_arrive(smem_u32(&bar[0]));
    }
    __syncthreads();
    Meetings meet;
    bool passed = true;
    if (threadIdx.x < 32) {
        passed = mbar_wait_warp(smem_u32(&bar[threadIdx.x & 1]), 0, &abort_flag, kSelftestCode, limit_ns);
        if (__any_sync(0xffffffffu, passed)) abort_flag = kSelftestParted;
    }
    if (passed) {
        if ((threadIdx.x & 31) == 0) done_with_step(nullptr, done, 2);
        meet.sync(1, 64);
        meet.sync(1, 64);
    }
    __syncwarp();
    meet.leave(1, 64, 2);
    __syncthreads();
    if (threadIdx.x == 0 && abort_flag != 0) *reinterpret_cast<volatile uint32_t*>(status) = abort_flag | ((uint32_t)blockIdx.x << 8);
}

}  // namespace fused

// What a wait that gave up leaves behind, and how the host takes note of it
struct WaitStatus {
    uint32_t* status = nullptr;    // status word, in page-locked host memory: the host reads it without a copy
    uint32_t* done_ctr = nullptr;  // see done_with_step
    cudaError_t create() {
        cudaError_t e = cudaMalloc((void**)&done_ctr, sizeof(uint32_t));
        if (e == cudaSuccess) e = cudaMemset(done_ctr, 0, sizeof(uint32_t));
        if (e == cudaSuccess) e = cudaHostAlloc((void**)&status, sizeof(uint32_t), cudaHostAllocPortable | cudaHostAllocMapped);
        if (e == cudaSuccess) *status = 0;
        return e;
    }
    // The kernels in question have been waited for.  Their warps that gave up may not have counted.
    unsigned take() {
        volatile uint32_t* word = status;
        const uint32_t v = *word;
        if (v != 0) {
            *word = 0;
            if (cudaMemset(done_ctr, 0, sizeof(uint32_t)) != cudaSuccess || cudaStreamSynchronize(nullptr) != cudaSuccess)
                cudaGetLastError();   // (a context that is gone; the caller reports the time-out)
        }
        return v;
    }
    void destroy() {
        if (status) cudaFreeHost(status);
        if (done_ctr) cudaFree(done_ctr);
    }
};

int fused_selftest_wait_timeout(unsigned limit_ms, unsigned* status_out) {
    WaitStatus w;
    cudaError_t e = w.create();
    if (e == cudaSuccess) {
        fused::k_selftest_wait_timeout<<<1, 64>>>(w.status, w.done_ctr, (unsigned long long)limit_ms * 1000000ull);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    uint32_t before = 0, after = 1;
    if (e == cudaSuccess) e = cudaMemcpy(&before, w.done_ctr, sizeof(before), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) *status_out = w.take();
    if (e == cudaSuccess) e = cudaMemcpy(&after, w.done_ctr, sizeof(after), cudaMemcpyDeviceToHost);
    w.destroy();
    if (e != cudaSuccess) return cuda_fail(e, "selftest", __FILE__, __LINE__);
    if (before != 1 || after != 0) {
        set_error("self-test: the count of a launch that gave up is %u, and %u after the check (1 and 0 expected)", before, after);
        return CFX_ERR_CUDA;
    }
    if ((*status_out & 0xFF) == fused::kSelftestParted) {
        set_error("self-test: some lanes of a warp went on from a wait that the others gave up");
        return CFX_ERR_CUDA;
    }
    return CFX_OK;
}

// ------------------------------------------------------------------ host side
struct FusedPlan {
    int device, n, H, L, A, precision;
    int game = CFX_GAME_FULL;
    uint8_t* image = nullptr;
    WaitStatus wait;
    float* state = nullptr;
    const float* params = nullptr;
    CUtensorMap state_map[fused::kMaxLayers];
    CUtensorMap quad_map[fused::kMaxLayers];   // the same with boxes of 32 rows
    CUtensorMap w_map[3];          // pair mode: operand image regions (encoder, gates, heads)
    CUtensorMap gate_map[2];       // tiles of 32 rows: see fused::Params
    int sm_count = 0;
    int pair = 0;        // 1: launch as clusters of two CTAs (cta_group::2 MMAs)
    int max_pairs = 0;   // co-resident clusters of two
    int max_split[2] = {0, 0};   // co-resident clusters of four and of two CTAs that share a tile
};

bool fused_supported(int H, int L, int A, int precision, int game) {
    const int want_a = game == CFX_GAME_CLASSIC ? fused::Gm<CFX_GAME_CLASSIC>::kA : fused::Gm<CFX_GAME_FULL>::kA;
    // hidden 256 for both games, hidden 128 for the full game
    const bool shape = H == 256 || (H == 128 && game == CFX_GAME_FULL);
    return shape && A == want_a && L >= 1 && L <= fused::kMaxLayers &&
           (precision == CFX_PREC_F16 || precision == CFX_PREC_BF16);
}

// kernel instantiation and its shared-memory size for (operand type, launch mode, game, hidden)
static const void* fused_kernel(int precision, int pair, int game, int H, bool rec16, int* smem) {
    const bool h = precision == CFX_PREC_F16;
#define CFX_K(T, P, G, HID)                                         \
    do {                                                            \
        *smem = fused::Cfg<P, G, HID>::kSmemBytes;                  \
        if constexpr (G == CFX_GAME_FULL)                           \
            if (rec16) return (const void*)fused::k_policy_fused<T, P, G, HID, true>; \
        return (const void*)fused::k_policy_fused<T, P, G, HID, false>; \
    } while (0)
#define CFX_K2(P, G, HID)                          \
    do {                                           \
        if (h) CFX_K(__half, P, G, HID);           \
        else CFX_K(__nv_bfloat16, P, G, HID);      \
    } while (0)
    if (game == CFX_GAME_CLASSIC) {
        if (pair) CFX_K2(true, CFX_GAME_CLASSIC, 256);
        CFX_K2(false, CFX_GAME_CLASSIC, 256);
    }
    if (H == 128) {
        if (pair) CFX_K2(true, CFX_GAME_FULL, 128);
        CFX_K2(false, CFX_GAME_FULL, 128);
    }
    if (pair) CFX_K2(true, CFX_GAME_FULL, 256);
    CFX_K2(false, CFX_GAME_FULL, 256);
#undef CFX_K2
#undef CFX_K
}

static size_t fused_image_bytes(int game, int H, int L) {
    if (game == CFX_GAME_CLASSIC) return fused::image_bytes<CFX_GAME_CLASSIC, 256>(L);
    return H == 128 ? fused::image_bytes<CFX_GAME_FULL, 128>(L) : fused::image_bytes<CFX_GAME_FULL, 256>(L);
}

int fused_create(FusedPlan** out, int device, int n, int H, int L, int A, int precision,
                 float* state, int game) {
    if (!fused_supported(H, L, A, precision, game)) {
        set_error("fused kernel: unsupported shape/precision");
        return CFX_ERR_UNSUPPORTED;
    }
    int major = 0, minor = 0, sm_count = 0;
    CFX_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device));
    CFX_CUDA(cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, device));
    CFX_CUDA(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device));
    if (major != 10) {
        set_error("fused kernel needs an sm_100 GPU (found sm_%d%d)", major, minor);
        return CFX_ERR_UNSUPPORTED;
    }
    FusedPlan* p = new FusedPlan();
    p->device = device; p->n = n; p->H = H; p->L = L; p->A = A; p->precision = precision;
    p->game = game;
    p->state = state;
    p->sm_count = sm_count;
    cudaError_t e = cudaMalloc((void**)&p->image, fused_image_bytes(game, H, L));
    if (e == cudaSuccess) e = p->wait.create();
    if (e != cudaSuccess) {
        fused_destroy(p);
        return cuda_fail(e, "fused_create alloc", __FILE__, __LINE__);
    }
    for (int l = 0; l < L; l++) {
        auto map = [&](CUtensorMap* m, int rows) {
            return make_tmap_2d(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, state + (size_t)l * n * H, (uint64_t)n, (uint64_t)H,
                                (uint64_t)H * 4, rows, fused::kHalfUnits, CU_TENSOR_MAP_SWIZZLE_128B);
        };
        if (!map(&p->state_map[l], fused::kTile) || !map(&p->quad_map[l], 32)) {
            fused_destroy(p);
            set_error("fused_create: cuTensorMapEncodeTiled failed for the state");
            return CFX_ERR_CUDA;
        }
    }
    for (int pr = 0; pr < 2 && e == cudaSuccess; pr++) {
        int smem = 0;
        for (int rec16 = 0; rec16 < 2 && e == cudaSuccess; rec16++) {
            const void* k = fused_kernel(precision, pr, game, H, rec16 != 0, &smem);
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        }
    }
    if (e != cudaSuccess) {
        fused_destroy(p);
        return cuda_fail(e, "cudaFuncSetAttribute", __FILE__, __LINE__);
    }
    // CTA pairs are the default (CFX_FUSED_PAIR=0 selects one CTA per tile); they need two
    // co-resident CTAs per cluster, otherwise the single-CTA kernel is used
    const char* pe = getenv("CFX_FUSED_PAIR");
    if (pe == nullptr || atoi(pe) != 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(2 * (unsigned)(p->sm_count / 2));
        cfg.blockDim = dim3(fused::kThreads);
        int smem = 0;
        const void* kpair = fused_kernel(precision, 1, game, H, false, &smem);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = 2; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
        cfg.attrs = &at; cfg.numAttrs = 1;
        int nc = 0;
        if (cudaOccupancyMaxActiveClusters(&nc, kpair, &cfg) == cudaSuccess && nc > 0) {
            p->pair = 1;
            p->max_pairs = nc;
        } else {
            cudaGetLastError();
        }
    }
    memset(p->w_map, 0, sizeof(p->w_map));
    memset(p->gate_map, 0, sizeof(p->gate_map));
    if (p->pair) {
        // The operand image seen as blocks of rows of 64 16-bit values (128 bytes), one tensor per region;
        // a box is what ONE CTA of a pair copies of a stage.  The image is already
        // swizzled, so the copies are not.
        const bool classic = game == CFX_GAME_CLASSIC;
        const int kblocks = H / 64;
        const int enc_blocks = classic ? fused::Gm<CFX_GAME_CLASSIC>::kEncBlocks : fused::Gm<CFX_GAME_FULL>::kEncBlocks;
        const int head_pair = classic ? fused::Gm<CFX_GAME_CLASSIC>::kHeadPair : fused::Gm<CFX_GAME_FULL>::kHeadPair;
        const uint64_t blocks[3] = {(uint64_t)enc_blocks, (uint64_t)L * (H / 64) * kblocks, 2};
        const uint64_t rows[3] = {(uint64_t)H, 3u * fused::kSliceUnits, (uint64_t)(kblocks * head_pair / 2)};
        const uint32_t box_blocks[3] = {256u / H, (uint32_t)kblocks, 1};
        const uint32_t box_rows[3] = {(uint32_t)H / 2, fused::kHalfRows / 2, (uint32_t)rows[2]};
        uint8_t* base = p->image;
        for (int r = 0; r < 3; r++) {
            if (!make_tmap_blocks(&p->w_map[r], base, blocks[r], rows[r], box_blocks[r], box_rows[r])) {
                fused_destroy(p);
                set_error("fused_create: cuTensorMapEncodeTiled failed for the operand image");
                return CFX_ERR_CUDA;
            }
            if (r == 1 && !(make_tmap_parts(&p->gate_map[0], base, blocks[r] * (fused::kSliceUnits / fused::kWarpUnits), 3, fused::kWarpUnits, 4, 2) &&
                            make_tmap_parts(&p->gate_map[1], base, blocks[r] * (fused::kSliceUnits / fused::kWarpUnits), 3, fused::kWarpUnits, 4, 1))) {
                fused_destroy(p);
                set_error("fused_create: cuTensorMapEncodeTiled failed for the gate blocks");
                return CFX_ERR_CUDA;
            }
            base += blocks[r] * rows[r] * 128;
        }
        for (int i = 0; i < 2; i++) {   // (the small-batch form reads the pairs' operand image)
            int rc = fused::split_prepare(precision, game, H, i == 0 ? 4 : 2, p->sm_count, &p->max_split[i]);
            if (rc) { fused_destroy(p); return rc; }
        }
    }
    *out = p;
    return CFX_OK;
}

int fused_refresh(FusedPlan* p, const float* params, cudaStream_t st) {
    p->params = params;
    const bool classic = p->game == CFX_GAME_CLASSIC;
    const ArenaLayout o = ArenaLayout::make(p->H, p->L, p->A, classic ? kClassicObs : kObs);
    const size_t total = fused_image_bytes(p->game, p->H, p->L) / 2;
    const unsigned blocks = (unsigned)((total + 255) / 256);
    const bool h = p->precision == CFX_PREC_F16;
#define CFX_PACK(T, G, HID) fused::k_pack_image<T, G, HID><<<blocks, 256, 0, st>>>(params, p->image, p->L, o.w_gru, o.w_a, o.w_v, p->pair)
    if (classic) { if (h) CFX_PACK(__half, CFX_GAME_CLASSIC, 256); else CFX_PACK(__nv_bfloat16, CFX_GAME_CLASSIC, 256); }
    else if (p->H == 128) { if (h) CFX_PACK(__half, CFX_GAME_FULL, 128); else CFX_PACK(__nv_bfloat16, CFX_GAME_FULL, 128); }
    else { if (h) CFX_PACK(__half, CFX_GAME_FULL, 256); else CFX_PACK(__nv_bfloat16, CFX_GAME_FULL, 256); }
#undef CFX_PACK
    CFX_CUDA(cudaGetLastError());
    return CFX_OK;
}

int fused_forward(FusedPlan* p, const FusedArgs& a, cudaStream_t st, int* launches) {
    if (a.r_state != nullptr && ((uintptr_t)a.r_state & 15) != 0) {
        set_error("fused forward: r_state must be 16-byte aligned");
        return CFX_ERR_INVALID;
    }
    if (a.logits_av != nullptr && ((uintptr_t)a.logits_av & 15) != 0) {
        set_error("fused forward: logits_av must be 16-byte aligned");
        return CFX_ERR_INVALID;
    }
    fused::Params P;
    const bool classic = p->game == CFX_GAME_CLASSIC;
    for (int l = 0; l < p->L; l++) P.state_map[l] = p->state_map[l];
    for (int r = 0; r < 3; r++) P.w_map[r] = p->w_map[r];
    for (int r = 0; r < 2; r++) P.gate_map[r] = p->gate_map[r];
    const ArenaLayout o = ArenaLayout::make(p->H, p->L, p->A, classic ? kClassicObs : kObs);
    P.records = a.records;
    P.state = a.state;
    P.image = p->image;
    P.params = p->params;
    P.prev_terminals = a.prev_terminals;
    P.uniforms = a.uniforms;
    P.env_actions = a.env_actions;
    P.actions = a.actions;
    P.logprobs = a.logprobs;
    P.values = a.values;
    P.logits_av = a.logits_av;
    P.r_state = a.r_state;
    P.r_state_bf16 = a.r_state_bf16;
    P.step_ctr = a.step_ctr;
    P.status = p->wait.status;
    P.done_ctr = p->wait.done_ctr;
    P.bump_step = a.bump_step;
    P.seed = a.seed;
    P.env_offset = a.env_offset;
    P.n = p->n;
    P.L = p->L;
    const int all_tiles = (p->n + fused::kTile - 1) / fused::kTile;
    P.tile_begin = a.tile_end > 0 ? a.tile_begin : 0;
    P.num_tiles = a.tile_end > 0 ? a.tile_end : all_tiles;
    // a CTA pair works on tiles 2c, 2c + 1: a slice must start at an even tile, and only the
    // slice that ends the batch may hold an odd number of tiles (its filler tile lies beyond n)
    if (P.tile_begin < 0 || P.num_tiles > all_tiles || P.tile_begin >= P.num_tiles || (P.tile_begin & 1) ||
        ((P.num_tiles & 1) && P.num_tiles != all_tiles)) {
        set_error("fused forward: bad tile range [%d, %d) of %d", P.tile_begin, P.num_tiles, all_tiles);
        return CFX_ERR_INVALID;
    }
    const int range_tiles = P.num_tiles - P.tile_begin;
    P.off_b_enc = o.b_enc;
    P.off_b_a = o.b_a;
    P.off_b_v = o.b_v;
    if (launches) *launches = 1;
    // Small batches: a tile is shared by four (two) CTAs as long as every tile then has its SMs at once, and is as
    // short as that allows (cfx_fused_split.cu).  CTAs of two slices take tiles of 64 and 128 rows; at 32 four CTAs a tile have their SMs.  With the 33
    // clusters of four and 74 of two that this part holds, four CTAs go to 1,056 and 2,112 envs, with 32 and 64 rows, and two to 4,736 with 64 rows and
    // 9,472 with 128.  At each of these limits the next form is slower, and the kernel below slower than all of them.  us a step, h256x2, clusters
    // of four with 32, 64, 128 rows, of two with 64 and 128, the kernel below: 1,056 envs 10.5, 14.6, 16.8, 16.2, 17.9, 21.5; 2,112 -, 14.8, 16.4, 16.5,
    // 18.2, 21.8; 4,224 -, -, 17.5, 16.9, 18.4, 22.0; 4,736 -, -, -, 17.1, 18.3, 22.3; 9,472 -, -, -, -, 19.0, 22.5.  h128x2, of two with 32, 64, 128 rows, the
    // kernel below: 2,368 envs 8.9, 12.5, 13.4, 15.7; 4,736 -, 12.9, 13.5, 15.7; 9,472 -, -, 14.0, 16.0.
    // From 2,113 to 4,224 envs four CTAs have 128 rows where write_r_state records the state in front of the cells, work that more CTAs share: the full game in fp32, or in
    // bf16 off a sector (four and two, us: h256x2 17.6 and 17.9, x4 26.4 and 27.5), and the classic game in fp32 from depth 3 on (x3 26.3 and 26.6).  Else two have 64:
    // without a record (4,224 envs h256x1 13.4 and 12.9, x3 21.5 and 20.7), with one that the cells write (x1 14.7 and 13.8, x3 23.2 and 22.1), in the classic
    // game (in bf16 x1 17.2 and 16.4, x3 26.0 and 25.4, in fp32 x2 22.0 and 21.4).
    const bool two_before_four = a.r_state == nullptr || (classic ? P.r_state_bf16 || p->L <= 2 : fused::record_by_rows(P));
    const int rows = std::min(p->n, P.num_tiles * fused::kTile) - P.tile_begin * fused::kTile;
    for (int i = 0; i < 2; i++)
        for (int S = i == 0 ? 4 : 2, tr = p->H == 64 * S ? 32 : 64; tr <= fused::kTile; tr *= 2) {
            const int tiles = (rows + tr - 1) / tr;
            if (tiles > p->max_split[i]) continue;
            if (S == 4 && tr == fused::kTile && two_before_four && (rows + 63) / 64 <= p->max_split[1]) continue;
            for (int l = 0; l < p->L; l++) P.state_map[l] = p->quad_map[l];
            P.tile_rows = tr;
            P.done_blocks = (uint32_t)(tiles * std::min(S, tr / 32));
            return fused::split_launch(p->precision, p->game, p->H, S, tiles, P, st);
        }
    int smem = 0;
    const void* kern = fused_kernel(p->precision, p->pair, p->game, p->H, fused::record_by_rows(P), &smem);
    void* kargs[1] = {(void*)&P};
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(fused::kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // see wait_for_previous_kernel
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    if (p->pair) {
        const int pairs = (range_tiles + 1) / 2;
        P.num_tiles_loop = P.tile_begin + 2 * pairs;
        cfg.gridDim = dim3(2u * (unsigned)(pairs < p->max_pairs ? pairs : p->max_pairs));
        at[1].id = cudaLaunchAttributeClusterDimension;
        at[1].val.clusterDim.x = 2; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
        cfg.numAttrs = 2;
    } else {
        P.num_tiles_loop = P.num_tiles;
        cfg.gridDim = dim3((unsigned)(range_tiles < p->sm_count ? range_tiles : p->sm_count));
    }
    P.done_blocks = cfg.gridDim.x;
    CFX_CUDA(cudaLaunchKernelExC(&cfg, kern, kargs));
    return CFX_OK;
}

unsigned fused_take_status(FusedPlan* p) { return p->wait.take(); }

void fused_destroy(FusedPlan* p) {
    if (!p) return;
    if (p->image) cudaFree(p->image);
    p->wait.destroy();
    delete p;
}

}  // namespace cfx
