// What the fused tcgen05 kernels share: shapes of the two games, layout of the operand image, launch
// parameters, operand types, record expansion, the MinGRU cell and the outputs of an env.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "cfx_common.cuh"
#include "cfx_f32x2.cuh"
#include "cfx_fused.h"
#include "cfx_sampler.cuh"
#include "cfx_tmap.h"
#include "cfx_umma.cuh"

namespace cfx {
using namespace umma;

namespace fused {

constexpr int kTile = 128;       // envs per tile
constexpr int kMaxLayers = 4;
constexpr int kSliceUnits = 64;  // hidden units per gate slice (N = 192: zh|zg|zp)
constexpr int kHalfUnits = 32;   // units of half a slice, and of a state box
constexpr int kHeadMax = 64;     // head accumulator columns reserved in tensor memory
// Shapes that follow from the hidden size the kernel is instantiated for (256 or 128).
template <int HID> struct Hd {
    static_assert(HID == 256 || HID == 128, "hidden sizes the kernel is built for");
    static constexpr int kH = HID;                        // hidden units
    static constexpr int kSlices = HID / kSliceUnits;     // gate slices per layer (4 / 2)
    static constexpr int kStateItems = HID / kHalfUnits;  // state boxes (128 rows x 32 units) per layer (8 / 4)
    static constexpr int kKBlocks = HID / 64;             // K blocks of 64 per HID-wide operand (4 / 2)
    static constexpr int kEncBlockBytes = HID * 128;      // one encoder block: [HID units][64 K] 16-bit
    static_assert((HID / 64) % 2 == 0, "a gate stage of one CTA per tile and a head slot of the small-batch form carry two K blocks");
};
// brings the shapes of Hd<HID> into a function body
#define CFX_DIMS(HID)                                                                        \
    constexpr int kH = Hd<HID>::kH, kSlices = Hd<HID>::kSlices, kStateItems = Hd<HID>::kStateItems, \
                  kKBlocks = Hd<HID>::kKBlocks;                                              \
    (void)kH; (void)kSlices; (void)kStateItems; (void)kKBlocks

// What differs between the two games the kernel is instantiated for.
//  full game (craftax_full.cu): 996-byte record = 792 map bytes + 51 raw floats, 843 features.
//    It is expanded by weight blocks (cfx_fused.cu) or in 16 chunks of 64 RECORD bytes (cfx_fused_split.cu): chunks 0-11 are 64
//    map bytes each (four K steps), chunk 12 is 24 map bytes and floats 0-9 (three K steps),
//    chunks 13 and 14 are 16 floats each and chunk 15 the last 9 floats (one K step each).  The
//    weight image has 14 blocks of 64 K columns: blocks 0-11 belong to chunks 0-11, block 12 to
//    chunks 12 and 13 (K columns 0-47 and 48-63), block 13 to chunks 14 and 15 (K columns 0-15
//    and 16-31).  43 actions;
//  classic game (craftax_classic.cu): 148-byte record, 1345 one-hot / scalar features in 22
//    chunks (one weight block each), 17 actions.
template <int GAME> struct Gm;
template <> struct Gm<CFX_GAME_FULL> {
    static constexpr int kA = 43, kEncChunks = 16, kEncBlocks = 14, kRecBytes = kRec;
    static constexpr int kHeadSingle = 48, kHeadPair = 64;   // head MMA N (pairs need N % 32 == 0)
};
template <> struct Gm<CFX_GAME_CLASSIC> {
    static constexpr int kA = 17, kEncChunks = 22, kEncBlocks = 22, kRecBytes = kClassicRec;
    static constexpr int kHeadSingle = 32, kHeadPair = 32;
};

// Image: blocks of 64 K columns, each a K-major, 128-byte-swizzled operand tile.  Encoder [block][HID units]; gate layers
// [layer][slice of 64 units][K block][192 rows], where the rows are zh|zg|zp of 16 units, the units that one worker warp
// handles, and then of the next 16: half of a slice is the 96 columns of one accumulator in cfx_fused.cu; heads.
constexpr int kGateBlockBytes = 3 * kSliceUnits * 128;               // block: [192 rows][64 K]
constexpr int kWarpUnits = 16;                                       // units of a slice that one worker warp handles
// row (accumulator column) of a gate (0 zh, 1 zg, 2 zp) of a slice's unit
__host__ __device__ constexpr int gate_row(int gate, int unit) { return (unit / kWarpUnits * 3 + gate) * kWarpUnits + unit % kWarpUnits; }
// head stage: one CTA per tile [K block][rows][64 K]; pairs [half][K block][rows / 2][64 K]
template <int GAME, int HID> __host__ __device__ constexpr int head_bytes(bool pair) {
    return Hd<HID>::kKBlocks * (pair ? Gm<GAME>::kHeadPair : Gm<GAME>::kHeadSingle) * 128;
}
template <int GAME, int HID> __host__ __device__ constexpr size_t enc_bytes() {
    return (size_t)Gm<GAME>::kEncBlocks * Hd<HID>::kEncBlockBytes;
}

template <int GAME, int HID> __host__ __device__ constexpr size_t image_bytes(int L) {   // room for either head layout
    return enc_bytes<GAME, HID>() + (size_t)L * Hd<HID>::kSlices * Hd<HID>::kKBlocks * kGateBlockBytes +
           (size_t)Hd<HID>::kKBlocks * kHeadMax * 128;
}

struct Params {
    // pair mode: the operand image as [blocks][rows][64] 16-bit tensors, one map per region (encoder,
    // gate layers, heads); a box is the part of a stage that one CTA of the pair copies
    CUtensorMap w_map[3];
    // small-batch form, tiles of 32 rows: the gate blocks as [16 units][gate][16 rows]; a box is zh and zg, or zp, of a slice
    CUtensorMap gate_map[2];
    CUtensorMap state_map[kMaxLayers];   // fp32 [n][256] per layer, box 128 x 32, SWIZZLE_128B
    const uint8_t* records;              // [n][996] (classic [n][148])
    const float* state;                  // [L][n][256]
    const uint8_t* image;                // pre-swizzled 16-bit weight blocks: see above
    const float* params;                 // fp32 arena (biases are read from it)
    const float* prev_terminals;
    const float* uniforms;
    float* env_actions;
    int32_t* actions;
    float* logprobs;
    float* values;
    float* logits_av;
    float* r_state;                      // optional [L][n][H] record of the post-zero input state
    int r_state_bf16;                    // the record holds bf16 instead of fp32
    unsigned long long* step_ctr;        // device step counter (Philox offset); see bump_step
    uint32_t* status;
    uint32_t* done_ctr;                  // blocks that are done with the step counter (bump_step)
    uint32_t done_blocks;                // how many there are (small-batch form: those that sample)
    int bump_step;
    uint64_t seed, env_offset;
    int n, L, num_tiles;  // num_tiles: end of the tile range of this launch (exclusive)
    int tile_begin;       // first tile of this launch (a launch may cover a slice of the envs)
    int tile_rows;        // small-batch form: rows of a tile
    int num_tiles_loop;   // trip bound of the tile loops: num_tiles, rounded up to even for CTA pairs
    size_t off_b_enc, off_b_a, off_b_v;
};

// ------------------------------------------------------------------ weight image
// Byte offset of (row, 16-bit K column c in [0,64)) inside a 128-byte-swizzled stage.
__host__ __device__ inline uint32_t sw128_off(uint32_t row, uint32_t byte_col) {
    return (row >> 3) * 1024 + (row & 7) * 128 + ((((byte_col >> 4) ^ (row & 7)) & 7) << 4) +
           (byte_col & 15);
}

// Feature behind K column c of encoder weight block `blk`, or -1 for padding.  Full game
// (feature kMap + i is raw float i of the record): blocks 0-11 map bytes 64 blk + c; block 12
// = map bytes 768-791, floats 0-9, 14 zero columns, floats 10-25; block 13 = floats 26-41,
// floats 42-50, zero columns.
template <int GAME> __host__ __device__ inline int enc_feature(int blk, int c) {
    if (GAME == CFX_GAME_CLASSIC) return blk * 64 + c < kClassicObs ? blk * 64 + c : -1;
    if (blk < 12) return blk * 64 + c;
    if (blk == 12) return c < 24 ? 768 + c : (c < 34 ? kMap + (c - 24) : (c < 48 ? -1 : kMap + 10 + (c - 48)));
    return c < 16 ? kMap + 26 + c : (c < 25 ? kMap + 42 + (c - 16) : -1);
}

// ------------------------------------------------------------------ small device helpers
template <typename T16>
struct Op16;
template <>
struct Op16<__half> {
    static constexpr uint32_t kFmt = kFmtF16;
    static constexpr uint32_t kOne = 0x3C00u;   // 1.0
    // two floats -> packed pair, `lo` in the low half (even K index)
    static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
        uint32_t r;
        asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
        return r;
    }
    static __device__ __forceinline__ float2 unpack(uint32_t v) {
        __half2 h = *reinterpret_cast<__half2*>(&v);
        return __half22float2(h);
    }
    // four record bytes (integers 0..255, exact in fp16) -> two packed pairs:
    // 0x6400 | b is the fp16 number 1024 + b; subtracting 1024 leaves b exactly.
    static __device__ __forceinline__ void bytes4(uint32_t w, uint32_t& p01, uint32_t& p23) {
        uint32_t a = __byte_perm(w, 0x64646464u, 0x5140);
        uint32_t b = __byte_perm(w, 0x64646464u, 0x7362);
        const uint32_t k = 0x64006400u;
        asm("sub.f16x2 %0, %1, %2;" : "=r"(p01) : "r"(a), "r"(k));
        asm("sub.f16x2 %0, %1, %2;" : "=r"(p23) : "r"(b), "r"(k));
    }
};
template <>
struct Op16<__nv_bfloat16> {
    static constexpr uint32_t kFmt = kFmtBF16;
    static constexpr uint32_t kOne = 0x3F80u;   // 1.0
    static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
        uint32_t r;
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
        return r;
    }
    static __device__ __forceinline__ float2 unpack(uint32_t v) {
        return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xFFFF0000u));
    }
    // 0x4B000000 | b is the fp32 number 2^23 + b; integers 0..255 are exact in bf16.
    static __device__ __forceinline__ void bytes4(uint32_t w, uint32_t& p01, uint32_t& p23) {
        const float m = 8388608.0f;
        float f0 = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440)) - m;
        float f1 = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7441)) - m;
        float f2 = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7442)) - m;
        float f3 = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7443)) - m;
        p01 = pack(f0, f1);
        p23 = pack(f2, f3);
    }
};

// MinGRU cell (k_mingru_epi_fwd, craftax_full.cu:9377-9381) with
// sigmoid(z) = 0.5 + 0.5 tanh(z/2) on the SFU and g(z) - 0.5 = max(z, 0.5 tanh(z/2))
// (equal to z for z >= 0 and to sigmoid(z) - 0.5 for z < 0).  The arguments are the HALVED
// pre-activations zh/2, zg/2, zp/2, which is what the gate MMAs produce (the operand image
// holds the gate weights times 0.5), so the cell starts with the tanh.
__device__ __forceinline__ float tanh_fast(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Two units at once with the packed fp32 instructions: the cell phase is bound by instruction
// issue and latency (four worker warps per scheduler), not by the FMA pipe.
// hzh, hzg, hzp: zh/2, zg/2, zp/2 of two units
__device__ __forceinline__ void mingru_cell_pair(float hzh0, float hzh1, float hzg0, float hzg1, float hzp0,
                                                 float hzp1, float st0, float st1, float x0, float x1,
                                                 float& out0, float& out1, float& h0, float& h1) {
    const uint64_t half2 = f2pack(0.5f, 0.5f), quarter2 = f2pack(0.25f, 0.25f), two2 = f2pack(2.0f, 2.0f);
    const uint64_t st = f2pack(st0, st1), x = f2pack(x0, x1);
    const uint64_t th = f2pack(tanh_fast(hzh0), tanh_fast(hzh1));
    const uint64_t tg = f2pack(tanh_fast(hzg0), tanh_fast(hzg1));
    const uint64_t tp = f2pack(tanh_fast(hzp0), tanh_fast(hzp1));
    const uint64_t sg = f2fma(tg, half2, half2), p = f2fma(tp, half2, half2);
    // g(zh) = 0.5 + max(zh, 0.5 th) = 0.5 + 2 max(zh/2, 0.25 th): every step is exact
    float m0, m1;
    f2unpack(f2mul(th, quarter2), m0, m1);
    const uint64_t gh = f2fma(two2, f2pack(fmaxf(hzh0, m0), fmaxf(hzh1, m1)), half2);
    const uint64_t out = f2fma(sg, f2sub(gh, st), st);
    const uint64_t h = f2fma(p, f2sub(out, x), x);
    f2unpack(out, out0, out1);
    f2unpack(h, h0, h1);
}

// ---------------------------------------------------------------- BPTT record of the state
// The optional record of the post-zero input state (what the reference's k_mingru_epi_fwd stores,
// craftax_full.cu:9370-9375), [L][n][H] fp32 or bf16.  A warp writes its 32 rows x 4 PIECES units from
// the state box (128-byte swizzled rows) before the cell updates it in place: PIECES lanes side by side take a row's
// 16-byte pieces, so that a store instruction touches 32 / PIECES rows.  With every lane writing the row whose cell
// it computes, it touched 32, and these stores kept the load/store unit busy for most of a slice (us in a loop over one set of
// buffers; over several in turn a step takes 3 to 7 % more): h256x2, 57,600 envs
// 126.6 -> 112.9 us with a bf16 record, 139.3 -> 123.1 with fp32; 16,416 envs 35.0 -> 30.7 and 37.1 -> 33.8; 8,192 envs
// (cfx_fused_split.cu) 25.9 -> 24.2 and 28.9 -> 25.2.
// `box`: the row of lane 0 (a multiple of 8 rows into the box); `at`: element of that row and the first of the warp's units
template <int PIECES, int HID>
__device__ __forceinline__ void write_r_state(const Params& P, const uint8_t* box, int piece0, size_t at, uint32_t zero_rows,
                                              int lane) {
    const int piece = lane % PIECES, k = lane / PIECES;
    // eight lanes in turn read shared memory without a bank conflict: rows that differ in bit 2 where they take two rows
    const int r0 = PIECES == 4 ? (k >> 1) | (k & 1) << 2 : k;
#pragma unroll
    for (int i = 0; i < PIECES; i++) {
        const int r = i * (32 / PIECES) + r0;
        float4 st = *reinterpret_cast<const float4*>(box + (r >> 3) * 1024 + (r & 7) * 128 + (((piece0 + piece) ^ (r & 7)) << 4));
        if (zero_rows >> r & 1u) st = make_float4(0.f, 0.f, 0.f, 0.f);
        const size_t o = at + (size_t)r * HID + 4 * piece;
        if (P.r_state_bf16)
            *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(P.r_state) + o) =
                make_uint2(Op16<__nv_bfloat16>::pack(st.x, st.y), Op16<__nv_bfloat16>::pack(st.z, st.w));
        else
            *reinterpret_cast<float4*>(P.r_state + o) = st;
    }
    __syncwarp();   // the cell's lanes overwrite the box
}

// The full game's bf16 record goes another way where it starts on a 32-byte sector: a thread's 16 units of its row are one sector, packed from the
// registers that the cell has its state in (REC16 kernels), so that nothing is read twice and no step of its own stands in front of the cell.  us a step,
// written by write_r_state and so: h256x2 9,504 envs 26.6 and 24.7, 37,888 70.6 and 65.8, 262,144 458 and 437; h128x2 16,416 19.0 and 17.7, 131,104 127 and 114;
// small batches h256x2 2,112 15.9 and 15.5, 6,400 21.9 and 21.3.  Slower, and not done so: fp32, two sectors a thread (h256x2 16,416 31.4 and 32.2);
// small batches of hidden 128 (9,472 15.0 and 15.5).  No difference in the classic game, which has no such kernels.
inline bool record_by_rows(const Params& P) { return P.r_state != nullptr && P.r_state_bf16 && (reinterpret_cast<uintptr_t>(P.r_state) & 31) == 0; }

// ------------------------------------------------------------------ record expansion
// One operand chunk (64 K columns, 32 packed pairs) of one env.
// Full game: chunk kc = record bytes [64 kc, 64 kc + 64) at `src` (4-byte aligned): map bytes, then raw
// floats; unused columns are zero.
template <typename Op>
__device__ __forceinline__ void expand_full(const uint8_t* src, int kc, uint32_t (&regs)[32]) {
    auto word = [&](int q) { return *reinterpret_cast<const uint32_t*>(src + 4 * q); };
    if (kc < 12) {          // 64 map bytes
#pragma unroll
        for (int q = 0; q < 16; q++) Op::bytes4(word(q), regs[2 * q], regs[2 * q + 1]);
    } else {
#pragma unroll
        for (int q = 0; q < 32; q++) regs[q] = 0u;
        if (kc == 12) {     // 24 map bytes, then raw floats 0-9
#pragma unroll
            for (int q = 0; q < 6; q++) Op::bytes4(word(q), regs[2 * q], regs[2 * q + 1]);
#pragma unroll
            for (int q = 0; q < 5; q++)
                regs[12 + q] = Op::pack(__uint_as_float(word(6 + 2 * q)), __uint_as_float(word(7 + 2 * q)));
        } else if (kc < 15) {   // 16 raw floats
#pragma unroll
            for (int q = 0; q < 8; q++)
                regs[q] = Op::pack(__uint_as_float(word(2 * q)), __uint_as_float(word(2 * q + 1)));
        } else {            // the last 9 raw floats; the record ends after them
#pragma unroll
            for (int q = 0; q < 4; q++)
                regs[q] = Op::pack(__uint_as_float(word(2 * q)), __uint_as_float(word(2 * q + 1)));
            regs[4] = Op::pack(__uint_as_float(word(8)), 0.0f);
        }
    }
}
// Weight block kc of the full game whole, from a record (chunks 12 and 13, 14 and 15 share one)
template <typename Op>
__device__ __forceinline__ void expand_block(const uint8_t* rec, int kc, uint32_t (&regs)[32]) {
    if (kc < 13) {
        expand_full<Op>(rec + 64 * kc, kc, regs);
        if (kc < 12) return;
    } else {
#pragma unroll
        for (int q = 0; q < 32; q++) regs[q] = 0u;
    }
    const float* f = reinterpret_cast<const float*>(rec + kMap);   // (4-byte aligned)
    if (kc == 12) {
#pragma unroll
        for (int q = 0; q < 8; q++) regs[24 + q] = Op::pack(f[10 + 2 * q], f[11 + 2 * q]);
    } else {
#pragma unroll
        for (int q = 0; q < 12; q++) regs[q] = Op::pack(f[26 + 2 * q], f[27 + 2 * q]);
        regs[12] = Op::pack(f[50], 0.0f);
    }
}
// K steps of 16 columns that chunk kc of the full game feeds
__host__ __device__ constexpr int full_ksteps(int kc) { return kc < 12 ? 4 : (kc == 12 ? 3 : 1); }

// Sixteen bits -> eight packed pairs of 1.0 / 0.0.  The even bits stay in the low half, the odd ones go one up in
// the high half; a mask then leaves one bit in each half, and one multiplication by 1.0's pattern, shifted down by
// the bits' position, makes both numbers (the patterns have enough low zeros for six positions).
template <typename Op>
__device__ __forceinline__ void bits16(uint32_t v, uint32_t* regs) {
    const uint32_t z0 = (v & 0x5555u) | ((v & 0xAAAAu) << 15), z1 = z0 >> 8;
    static_assert((Op::kOne & 0x3Fu) == 0, "shifts are exact");
#pragma unroll
    for (int q = 0; q < 4; q++) {
        regs[q] = (z0 & (0x00010001u << 2 * q)) * (Op::kOne >> 2 * q);
        regs[4 + q] = (z1 & (0x00010001u << 2 * q)) * (Op::kOne >> 2 * q);
    }
}
// Classic game: the 1323 one-hot features of a record (148 bytes at `rp`) are a bit stream, 21 bits per
// view cell (17 block ids + 4 mob bits); a chunk is a 64-bit window of it, built from at most four
// cells, and every bit becomes 1.0 or 0.0.  Chunk 20 ends with the 21 scalar features
// (feature order of expand_obs_kernel, craftax_classic.cu:1265-1301), chunk 21 holds the sleeping flag alone.
template <typename Op>
__device__ __forceinline__ void expand_classic(const uint8_t* rp, int kc, uint32_t (&regs)[32]) {
    constexpr int kEncChunks = Gm<CFX_GAME_CLASSIC>::kEncChunks;
    auto cell_bits = [&](int cell) -> uint64_t {
        if (cell >= kClassicCells) return 0ull;
        const uint32_t blk = rp[cell], mob = rp[kClassicCells + cell];
        return (uint64_t)((blk < (uint32_t)kClassicBlocks ? (1u << blk) : 0u) | ((mob & 15u) << kClassicBlocks));
    };
    const int cell0 = (64 * kc) / 21, off0 = 64 * kc - 21 * cell0;
    uint64_t w = 0;
    if (kc < kEncChunks - 1)
        w = (cell_bits(cell0) >> off0) | (cell_bits(cell0 + 1) << (21 - off0)) |
            (cell_bits(cell0 + 2) << (42 - off0)) | (cell_bits(cell0 + 3) << (63 - off0));
    const uint32_t wlo = (uint32_t)w, whi = (uint32_t)(w >> 32);
    bits16<Op>(wlo, regs);
    bits16<Op>(wlo >> 16, regs + 8);
    bits16<Op>(whi, regs + 16);
    bits16<Op>(whi >> 16, regs + 24);
    if (kc == kEncChunks - 2) {   // features 1280..1343: 43 one-hot bits, then 21 scalars
        float sc[22];
#pragma unroll
        for (int j2 = 0; j2 < 16; j2++) sc[j2] = (float)(int8_t)rp[2 * kClassicCells + j2] / 10.0f;
        const int dir = (int8_t)rp[2 * kClassicCells + 16];
#pragma unroll
        for (int d = 0; d < 4; d++) sc[16 + d] = dir == d + 1 ? 1.0f : 0.0f;
        sc[20] = *reinterpret_cast<const float*>(rp + 2 * kClassicCells + 18);
        sc[21] = 0.0f;
        regs[21] = (regs[21] & 0xFFFFu) | (Op::pack(0.0f, sc[0]) & 0xFFFF0000u);
#pragma unroll
        for (int q = 22; q < 32; q++) regs[q] = Op::pack(sc[2 * (q - 22) + 1], sc[2 * (q - 22) + 2]);
    } else if (kc == kEncChunks - 1) {   // feature 1344: sleeping
        regs[0] = rp[2 * kClassicCells + 17] != 0 ? Op::kOne : 0u;
    }
}

// ------------------------------------------------------------------ step counter
// The reference bumps the sampler offset with a one-thread kernel after the step (k_bump_ctr, craftax_full.cu:12085).  Here
// the last of `readers` to say that it has read the counter raises it.  A launch in which one gave up before it came to that
// leaves the count where it is: WaitStatus::take clears it.
__device__ __forceinline__ void done_with_step(unsigned long long* step, uint32_t* done, uint32_t readers) {
    __threadfence();
    if (atomicAdd(done, 1u) == readers - 1) {
        *step += 1ULL;
        *done = 0u;
    }
}

// ------------------------------------------------------------------ meetings of worker warps
// The named barriers at which a warp meets others of its block: id `first`, then the one after it, each once a launch.  A
// named barrier has no limit, so a warp that gives up in a bounded wait before a meeting arrives there
// on its way out (leave): nobody waits for a warp that has gone.  (Only `met` lives through the role, and what a warp that
// gave up still owes is worked out for such a warp alone: 4,000 envs 19.5 us so, 19.85 with every warp working it out.  The
// check itself costs the smallest batches 1 %, 1,024 envs 12.7 us instead of 12.6; where the waits give up instead: 12.8.)
struct Meetings {
    static constexpr int kAll = 255;   // the role has come to its end
    int met = 0;
    __device__ __forceinline__ void sync(int first, int threads) {
        asm volatile("bar.sync %0, %1;" ::"r"(first + met), "r"(threads) : "memory");
        met++;
    }
    __device__ __forceinline__ void arrive(int first, int threads) {
        asm volatile("bar.arrive %0, %1;" ::"r"(first + met), "r"(threads) : "memory");
        met++;
    }
    __device__ __forceinline__ void leave(int first, int threads, int meetings) {
        while (met < meetings) arrive(first, threads);
    }
};

// ------------------------------------------------------------------ outputs of an env
template <int GAME, int A>
__device__ __forceinline__ void write_logits(const Params& P, int env, const float (&logits)[A], float value) {
    constexpr int kA = Gm<GAME>::kA;
    static_assert(A == kA, "actions");
    if constexpr ((kA + 1) % 8 != 4) {
        static_assert((kA + 1) % 2 == 0, "rows are 8-byte aligned");
        float* dst = P.logits_av + (size_t)env * (kA + 1);
        if (P.logits_av != nullptr) {
#pragma unroll
            for (int a = 0; a < kA + 1; a += 2)
                *reinterpret_cast<float2*>(dst + a) = make_float2(logits[a], a + 1 < kA ? logits[a + 1 < kA ? a + 1 : a] : value);
        }
    } else if (P.logits_av != nullptr) {
        // A row is 176 bytes: 32-byte aligned for every other env, 16 bytes off for the
        // ones between.  It goes out as five 32-byte stores and one 16-byte store (in
        // front for the rows that are off, at the end for the others): whole sectors, and 6 store
        // instructions per warp instead of 11.  (The store burst of the sampler
        // holds up every shared-memory and barrier operation of the SM behind it.)
        constexpr int kRow = kA + 1;
        static_assert(kRow % 8 == 4, "row = five 32-byte pieces and one 16-byte piece");
        float rowv[kRow];
#pragma unroll
        for (int a = 0; a < kA; a++) rowv[a] = logits[a];
        rowv[kA] = value;
        float* dst = P.logits_av + (size_t)env * kRow;
        // (the array itself need only be 16-byte aligned: what counts is the row's address)
        const bool odd = (reinterpret_cast<uintptr_t>(dst) & 31u) != 0;
        float4 v4;
        v4.x = odd ? rowv[0] : rowv[kRow - 4];
        v4.y = odd ? rowv[1] : rowv[kRow - 3];
        v4.z = odd ? rowv[2] : rowv[kRow - 2];
        v4.w = odd ? rowv[3] : rowv[kRow - 1];
        *reinterpret_cast<float4*>(dst + (odd ? 0 : kRow - 4)) = v4;
#pragma unroll
        for (int q = 0; q < kRow / 8; q++) {
            float v8[8];
#pragma unroll
            for (int e = 0; e < 8; e++) v8[e] = odd ? rowv[8 * q + 4 + e] : rowv[8 * q + e];
            st_global_v8(dst + 8 * q + (odd ? 4 : 0), v8);
        }
    }
}
__device__ __forceinline__ void write_action(const Params& P, int env, int act, float lp, float value) {
    if (P.env_actions) P.env_actions[env] = (float)act;
    P.actions[env] = act;
    if (P.logprobs) P.logprobs[env] = lp;
    if (P.values) P.values[env] = value;
}
// Head accumulator row + biases (bias[a] for action a, bias[kA] for the value) -> logits_av, sampled
// action, log-probability, value.
template <int GAME, int N>
__device__ __forceinline__ void write_outputs(const Params& P, int env, const uint32_t (&hv)[N], const float* bias, float u) {
    constexpr int kA = Gm<GAME>::kA;
    static_assert(N > kA, "columns");
    float logits[kA];
#pragma unroll
    for (int a = 0; a < kA; a++) logits[a] = __uint_as_float(hv[a]) + bias[a];
    const float value = __uint_as_float(hv[kA]) + bias[kA];
    write_logits<GAME>(P, env, logits, value);
    float lp;
    const int act = sample_action<kA>(logits, u, &lp);
    write_action(P, env, act, lp, value);
}

}  // namespace fused
}  // namespace cfx
