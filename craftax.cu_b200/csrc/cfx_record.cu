// Record write: env state -> 996-byte compact records (reference k_record_obs /
// cf_record_env_warp, craftax_full.cu:9180-9297; scalar tail :2429-2487).
//
// The reference gives every env a warp and lets lane 0 walk the mob slots and compute the 51
// tail scalars; every one of its ~110 scalar loads then fetches 4 bytes of a sector on its own,
// one after the other.  Here a block of eight warps owns 32 consecutive envs:
//   1. lane per env: position, level and flag; then, all of a lane's in flight, the ~50 SoA fields and the 14 mob slots of
//      the player's level, lane e for env e, so that a warp's loads of a field are one 128-byte line, each warp an eighth of
//      them (Gather);
//   2. under these loads, the copies of the views to shared memory: in each of three map planes 9 rows of 11 bytes, 48 bytes apart.
//      A warp copies the 395 bytes from first to last row of a plane side by side, an instruction a plane and env, for its four envs;
//      then the fields become the 51 tail floats, and the mobs (an earlier slot of a class that a later slot covers is dropped) go
//      to shared memory;
//   3. warp per env: a lane makes four cells of a view row from the spans in registers, the four records
//      are put together where the spans were, and go out as one bulk copy (1,992 blocks of 16 bytes a
//      block) or, where an env is skipped, as coalesced words.
// 65,536 envs with 62 KB of maps each: 38.4 us, with the list of 250 reset envs behind it 44.6; 128 MB read from DRAM.  What it gained (us, by itself; with the
// list): loads that wait for nothing in front of the copies 46.4 -> 42.5, 52.9 -> 49.1; whole spans for rows piece by piece 41.8, 48.0; the fields in front of
// what depends on the level 39.9, 46.2; 64 bytes a miss (ld_bits) 38.4, 44.6.  A block took 25,000 cycles and takes 17,000; the memory latencies one behind
// the other, 8,000 of them, are left.
// The bytes are the reference's: the same predicates, the same "last slot of a class wins a
// cell" order, the same float expressions (sqrtf(x) * 0.1f, x * 0.1f, x * 0.5f, x * 0.25f; no
// fused multiply-add can form).
#include <cuda_runtime.h>

#include <cstddef>
#include <type_traits>

#include "cfx_common.cuh"

namespace cfx {
namespace record {

constexpr int kRows = 9, kCols = 11;   // view around the player
constexpr int kMapSize = 48, kLevels = 9, kMobTypes = 8, kClasses = 5, kSlots = 3;
constexpr int kMobs = kClasses * kSlots;                       // slot 2 of class 2 is never used
constexpr int kLit = 12;                                       // light_map > 12 = visible
constexpr int kKilledToClear = 8;
constexpr int kBlockEnvs = 32, kBlockThreads = 256;

struct Params {
    cfx_env_view v;
    uint8_t* records;
    const uint8_t* skip;
    const uint8_t* list;
    int list_stride;
    const int* count_dev;
    int n;
};
// The view in a plane: nine rows of eleven bytes, 48 apart, so 395 bytes from the first to the last, in 26 pieces of 16
constexpr int kPlanes = 3, kSpan = kRows * kMapSize, kPieces = 26;
constexpr int kRowWords = (3 + kCols + 3) / 4;   // that a view row lies in
static_assert(15 + (kRows - 1) * kMapSize + kCols <= 16 * kPieces && 16 * kPieces <= kSpan && kPieces <= 32, "a lane a piece");
constexpr int kWarps = kBlockThreads / 32, kOwn = kBlockEnvs / kWarps;   // envs whose records a warp writes
constexpr int kPlaneBytes = kMapSize * kMapSize, kRecWords = kRec / 4, kMapWords = kMap / 4;
struct Gathered {
    float tail[kBlockEnvs][kTail];       // odd row length: conflict-free thread-per-env writes
    uint32_t mobs[kBlockEnvs][kMobs];
};
struct Shared : Gathered {
    // per warp its four records as they go out, and before that, until they are in registers, the spans of its four
    // envs' views (light, block, item)
    __align__(16) uint8_t span[kWarps][kOwn * kPlanes * kSpan];
};
static_assert(kOwn * kRec % 16 == 0 && kRec <= kPlanes * kSpan && kSpan % 16 == 0, "a warp's records are whole 16-byte words");

// craftax_wg_jax_index (:1963-1975): negative indices wrap once, then clamp
__device__ __forceinline__ int jax_index(int i, int size) {
    if (i < 0) i += size;
    if (i < 0) return 0;
    return i >= size ? size - 1 : i;
}
// Loads that are issued where they stand.  A plain load through a pointer of the view may alias the shared memory
// that is written in between, so the compiler keeps load, conversion and store of every field in order, one DRAM
// latency a field; a read-only load it sinks to its use, with the same effect.  Every loop below
// therefore loads all its fields first.  (ld.global.nc would be wrong besides: see wait_for_previous_kernel.)
// What a miss brings into L2 is limited to 64 bytes, a burst of the memory, here and in the copies: an env on another level than its neighbours reads
// scattered words, and a view's span ends anywhere.  By default more comes along (us: this kernel and its list 46.1 -> 44.6; classic game, 262,144 envs 27.4 -> 25.8, its
// reads from memory 102 -> 86 MB).  Not for bytes and shorts, of whose burst the neighbouring blocks use the rest (classic 27.2 -> 27.5).  The words past L1:
// 65,536 envs 0.4 % faster, but lanes and warps read the same lines: 4,096 envs 8.6 -> 10.0, a list of 1,000 of 65,536 4.4 -> 5.9.
__device__ __forceinline__ uint32_t ld_bits(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.L2::64B.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int32_t ld_now(const int32_t* p) { return (int32_t)ld_bits(reinterpret_cast<const uint32_t*>(p)); }
__device__ __forceinline__ uint32_t ld_now(const uint32_t* p) { return ld_bits(p); }
__device__ __forceinline__ float ld_now(const float* p) { return __uint_as_float(ld_bits(reinterpret_cast<const uint32_t*>(p))); }
__device__ __forceinline__ uint8_t ld_now(const uint8_t* p) {
    uint16_t v;
    asm volatile("ld.global.u8 %0, [%1];" : "=h"(v) : "l"(p));
    return (uint8_t)v;
}
__device__ __forceinline__ int8_t ld_now(const int8_t* p) { return (int8_t)ld_now(reinterpret_cast<const uint8_t*>(p)); }
__device__ __forceinline__ int16_t ld_now(const int16_t* p) {
    int16_t v;
    asm volatile("ld.global.s16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}
template <typename T>
__device__ __forceinline__ T soa(const T* f, int elem, int n, int e) {
    return ld_now(f + ((size_t)elem * (size_t)n + (size_t)e));
}
// flat index of (class, level, slot) in the mob fields (CFM, :715)
__device__ __forceinline__ int mob_index(int c, int level, int i) { return (c * kLevels + level) * kSlots + i; }

// a mob inside the view and on the map: valid | cell << 8 | channel << 4 | value
__device__ __forceinline__ uint32_t pack_mob(int c, int type_id, bool mask, int mr, int mc, int top, int left) {
    const int lr = mr - top, lc = mc - left;
    const bool on = type_id >= 0 && type_id < kMobTypes && mask && lr >= 0 && lr < kRows && lc >= 0 && lc < kCols &&
                    mr >= 0 && mr < kMapSize && mc >= 0 && mc < kMapSize;
    return on ? 0x80000000u | (uint32_t)(lr * kCols + lc) << 8 | (uint32_t)(3 + c) << 4 | (uint32_t)(type_id + 1) : 0u;
}
__device__ __forceinline__ bool same_cell(uint32_t a, uint32_t b) {
    return (a & b & 0x80000000u) && ((a ^ b) & 0xFF00u) == 0;
}

// The kN slots of a mob class c on a level: which are alive, then what and where those are, then the slots as they go into the record
template <int kN> struct Mobs {
    uint8_t on[kN];
    int32_t type[kN], row[kN], col[kN];
    __device__ __forceinline__ void load_alive(const cfx_env_view& V, int e, int c, int mob_level) {
#pragma unroll
        for (int i = 0; i < kN; i++) on[i] = soa(V.mob_mask, mob_index(c, mob_level, i), V.num_envs, e);
    }
    // only where a mob is alive: an env on another level than its neighbours reads a 64-byte burst for every word
    __device__ __forceinline__ void load_slots(const cfx_env_view& V, int e, int c, int mob_level) {
#pragma unroll
        for (int i = 0; i < kN; i++) {
            const int idx = mob_index(c, mob_level, i);
            type[i] = row[i] = col[i] = -1;
            if (on[i] != 0) {
                type[i] = soa(V.mob_type_id, idx, V.num_envs, e);
                row[i] = soa(V.mob_position, idx * 2, V.num_envs, e);
                col[i] = soa(V.mob_position, idx * 2 + 1, V.num_envs, e);
            }
        }
    }
    __device__ __forceinline__ bool put(int c, int top, int left, uint32_t* mobs) const {   // true if one is alive
        bool alive = false;
        uint32_t pk[kSlots] = {0, 0, 0};
#pragma unroll
        for (int i = 0; i < kN; i++) {
            alive = alive || on[i] != 0;
            pk[i] = pack_mob(c, type[i], on[i] != 0, row[i], col[i], top, left);
        }
        // "last slot wins": a later slot of the class on the same cell replaces an earlier one
        // (:9222-9231); the earlier one is dropped here, so the stores of phase 3 need no order
#pragma unroll
        for (int i = 0; i < kN - 1; i++)
#pragma unroll
            for (int i2 = i + 1; i2 < kN; i2++)
                if (same_cell(pk[i], pk[i2])) pk[i] = 0;
#pragma unroll
        for (int i = 0; i < kSlots; i++) mobs[c * kSlots + i] = pk[i];
        return alive;
    }
};

// phase 2: everything of env e that does not depend on the cell.  Lane t of EVERY warp of the block works on env t of
// the block; warp `part` takes an eighth of the loads.  The 51 scalars are in the order of
// craftax_encode_scalar_observation_tail_at (:2429-2487).  In three steps, each a memory latency: the fields, which wait for nothing; what depends on
// the level; the mobs that are alive.  (All of it behind the copies of the map rows, and the two classes of part 4 one after the other,
// made that warp the last of the block by 5,000 of its 25,000 cycles.)
struct Gather {
    uint32_t raw[13];
    int32_t killed;
    Mobs<kSlots> first;   // of class 0 in part 4, of classes 1, 3 and 4 in parts 5 to 7
    Mobs<2> ranged;       // of class 2, whose third slot is never used, in part 4
    __device__ __forceinline__ void load_fields(const cfx_env_view& V, int e, int part) {
        const int n = V.num_envs;
        auto word = [&](const auto* f, int elem) { return ld_bits(reinterpret_cast<const uint32_t*>(f) + ((size_t)elem * (size_t)n + (size_t)e)); };
        if (part == 0) {
            const int32_t* const f[12] = {V.inv_wood, V.inv_stone, V.inv_coal, V.inv_iron, V.inv_diamond, V.inv_sapphire,
                                          V.inv_ruby, V.inv_sapling, V.inv_torches, V.inv_arrows, V.inv_books, V.inv_pickaxe};
#pragma unroll
            for (int i = 0; i < 12; i++) raw[i] = word(f[i], 0);
        } else if (part == 1) {
            const int32_t* const f[4] = {V.inv_sword, V.sword_enchantment, V.bow_enchantment, V.inv_bow};
#pragma unroll
            for (int i = 0; i < 4; i++) raw[i] = word(f[i], 0);
#pragma unroll
            for (int i = 0; i < 6; i++) raw[4 + i] = word(V.inv_potions, i);
            raw[10] = word(V.player_health, 0);
        } else if (part == 2) {
            const int32_t* const f[9] = {V.player_food, V.player_drink, V.player_energy, V.player_mana, V.player_xp,
                                         V.player_dexterity, V.player_strength, V.player_intelligence, V.player_direction};
#pragma unroll
            for (int i = 0; i < 9; i++) raw[i] = word(f[i], 0);
#pragma unroll
            for (int i = 0; i < 4; i++) raw[9 + i] = word(V.inv_armour, i);
        } else if (part == 3) {
#pragma unroll
            for (int i = 0; i < 4; i++) raw[i] = word(V.armour_enchantments, i);
            raw[4] = word(V.light_level, 0);
            raw[5] = soa(V.is_sleeping, 0, n, e);
            raw[6] = soa(V.is_resting, 0, n, e);
            raw[7] = soa(V.learned_spells, 0, n, e);
            raw[8] = soa(V.learned_spells, 1, n, e);
        } else if (part == 4) {
            raw[0] = word(V.boss_timesteps_to_spawn_this_round, 0);
        }
    }
    // mobs of the player's level inside the view and on the map (:9195-9236).  Whether the cell is lit is
    // looked up in the copied row when the record is put together: two slots on one cell are both lit or
    // both not, so the order of dropping does not depend on it.
    __device__ __forceinline__ void load_of_level(const cfx_env_view& V, int e, int part, int level) {
        const int mob_level = jax_index(level, kLevels);
        if (part == 3) {
            killed = soa(V.monsters_killed, (unsigned)level < (unsigned)kLevels ? level : 0, V.num_envs, e);
        } else if (part >= 4) {
            first.load_alive(V, e, mob_class(part), mob_level);
            if (part == 4) ranged.load_alive(V, e, 2, mob_level);
        }
    }
    __device__ __forceinline__ void finish(const cfx_env_view& V, int e, int t, int part, int level, int top, int left, Gathered& S) {
        const int mob_level = jax_index(level, kLevels);
        float* o = S.tail[t];
        auto whole = [&](int i) { return (float)(int32_t)raw[i]; };
        if (part == 0) {
#pragma unroll
            for (int i = 0; i < 10; i++) o[i] = sqrtf(whole(i)) * (1.0f / 10.0f);
            o[10] = whole(10) * (1.0f / 2.0f);
            o[11] = whole(11) * (1.0f / 4.0f);
        } else if (part == 1) {
            o[12] = whole(0) * (1.0f / 4.0f);
#pragma unroll
            for (int i = 0; i < 3; i++) o[13 + i] = whole(1 + i);
#pragma unroll
            for (int i = 0; i < 6; i++) o[16 + i] = sqrtf(whole(4 + i)) * (1.0f / 10.0f);
            o[22] = __uint_as_float(raw[10]) * (1.0f / 10.0f);
        } else if (part == 2) {
#pragma unroll
            for (int i = 0; i < 8; i++) o[23 + i] = whole(i) * (1.0f / 10.0f);
            const int direction_index = (int)raw[8] - 1;
#pragma unroll
            for (int i = 0; i < 4; i++) o[31 + i] = i == direction_index ? 1.0f : 0.0f;
#pragma unroll
            for (int i = 0; i < 4; i++) o[35 + i] = whole(9 + i) * (1.0f / 2.0f);
        } else if (part == 3) {
#pragma unroll
            for (int i = 0; i < 4; i++) o[39 + i] = whole(i);
            o[43] = __uint_as_float(raw[4]);
#pragma unroll
            for (int i = 0; i < 4; i++) o[44 + i] = raw[5 + i] != 0 ? 1.0f : 0.0f;
            o[48] = (float)level * (1.0f / 10.0f);
            o[49] = (unsigned)level < (unsigned)kLevels && killed >= kKilledToClear ? 1.0f : 0.0f;
        } else {
            const int c = mob_class(part);
            first.load_slots(V, e, c, mob_level);
            if (part == 4) ranged.load_slots(V, e, 2, mob_level);
            const bool alive = first.put(c, top, left, S.mobs[t]);
            // craftax_wg_is_boss_vulnerable (:1988-2003): no melee and no ranged mob alive on the level
            if (part == 4) o[50] = !ranged.put(2, top, left, S.mobs[t]) && !alive && (int32_t)raw[0] <= 0 ? 1.0f : 0.0f;
        }
    }
private:
    static __device__ __forceinline__ int mob_class(int part) { return part == 4 ? 0 : part == 5 ? 1 : part - 3; }
};

// What the copies and the assembly of one env need, in a word: top and left of the view, plane of the level, and whether there
// is such a level.
struct View {
    uint32_t bits;   // (top + 32) | (left + 32) << 8 | plane << 16 | ok << 24
    __device__ __forceinline__ int top() const { return (int)(bits & 255u) - 32; }
    __device__ __forceinline__ int left() const { return (int)(bits >> 8 & 255u) - 32; }
    __device__ __forceinline__ int level() const { return bits >> 16 & 255u; }
    __device__ __forceinline__ bool level_ok() const { return bits >> 24; }
};
__device__ __forceinline__ View make_view(int level, int top, int left) {
    top = min(max(top, -32), 64);      // (a view that is off the map stays off it)
    left = min(max(left, -32), 64);
    return {(uint32_t)(top + 32) | (uint32_t)(left + 32) << 8 | (uint32_t)jax_index(level, kLevels) << 16 |
            ((unsigned)level < (unsigned)kLevels ? 1u << 24 : 0u)};
}
// Where byte `o` of view row dr lies in a span, counted from the 16-byte word of the view's first byte; the nine rows start in eight
// different groups of four banks
__device__ __forceinline__ int row_byte(int dr, int o) { return dr * kMapSize + o; }
// The part of a lane in the copies of an env's view (light, block, item)
struct CopyLane {
    int lane;
    __device__ __forceinline__ explicit CopyLane(int l) : lane(l) {}
    // Planes that are not aligned to words: a lane takes every 32nd cell of the view, its bytes of the three planes all in flight
    // (65,536 envs 55 us; 75 with the bytes of a row one after the other)
    __device__ __forceinline__ void bytes(const cfx_env_view& V, int e, View v, uint8_t* dst) const {
        constexpr int kCells = kRows * kCols, kRounds = (kCells + 31) / 32;
        const uint64_t off[kPlanes] = {V.light_map_offset, V.map_offset, V.item_map_offset};
        const uint8_t* q = V.state_base + (size_t)e * V.state_stride + v.level() * kPlaneBytes;
        uint8_t b[kRounds][kPlanes];
#pragma unroll
        for (int i = 0; i < kRounds; i++) {
            const int cell = lane + 32 * i, row = v.top() + cell / kCols, col = v.left() + cell % kCols;
            const bool in = cell < kCells && (unsigned)row < (unsigned)kMapSize && (unsigned)col < (unsigned)kMapSize;
#pragma unroll
            for (int p = 0; p < kPlanes; p++) b[i][p] = in ? ld_now(q + off[p] + row * kMapSize + col) : (uint8_t)0;
        }
#pragma unroll
        for (int i = 0; i < kRounds; i++) {
            const int cell = lane + 32 * i;
            if (cell >= kCells) break;
#pragma unroll
            for (int p = 0; p < kPlanes; p++) dst[p * kSpan + row_byte(cell / kCols, (v.left() & 15) + cell % kCols)] = b[i][p];
        }
    }
    // Starts the copies of env e's view into `dst`: where the planes are aligned to 16 bytes, the pieces of a plane's span side by
    // side, an instruction a plane (what lies between the view's rows comes along: memory is read in bursts of 64 bytes anyway);
    // else the words that the view's rows lie in, four lanes a row (eight rows are 32 banks).  Words, us: a lane a row, its words one instruction
    // after the other, 65,536 envs 50.7, 1,000 5.51, a list of all envs 55.8; so 48.9, 5.37, 54.4.  Bytes: 55.1, 6.39, 74.2.
    template <bool BYTES>
    __device__ __forceinline__ void start(const cfx_env_view& V, int e, View v, int grain, uint8_t* dst) const {
        if constexpr (BYTES) return bytes(V, e, v, dst);
        const uint64_t off[kPlanes] = {V.light_map_offset, V.map_offset, V.item_map_offset};
        const uint8_t* const q = V.state_base + (size_t)e * V.state_stride + v.level() * kPlaneBytes;
        const int left = v.left(), c0 = left & ~15;
        if (grain == 16) {
            const int at = v.top() * kMapSize + c0 + 16 * lane;
            if (lane >= kPieces || (unsigned)at >= (unsigned)kPlaneBytes) return;
#pragma unroll
            for (int p = 0; p < kPlanes; p++)
                asm volatile("cp.async.cg.shared.global.L2::64B [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + p * kSpan + 16 * lane)), "l"(q + off[p] + at) : "memory");
        } else {
            static_assert(kRowWords == 4 && kRows == 9, "eight rows an instruction, and the last one of the three planes");
            const int o = (left & 12) + 4 * (lane & 3), col = c0 + o, dr = lane >> 2, row = v.top() + dr, last = v.top() + 8;
            if ((unsigned)col >= (unsigned)kMapSize || col >= left + kCols) return;
            auto word = [&](int p, uint64_t plane, int r, int at) {
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + p * kSpan + row_byte(r, o))), "l"(q + plane + (at * kMapSize + col)) : "memory");
            };
            if ((unsigned)row < (unsigned)kMapSize)
#pragma unroll
                for (int p = 0; p < kPlanes; p++) word(p, off[p], dr, row);
            if (dr < kPlanes && (unsigned)last < (unsigned)kMapSize) word(dr, dr == 0 ? off[0] : dr == 1 ? off[1] : off[2], 8, last);
        }
    }
};
__device__ __forceinline__ void wait_spans() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncwarp();
}
__host__ __device__ __forceinline__ int copy_grain(const cfx_env_view& V) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(V.state_base) | V.state_stride | V.map_offset | V.item_map_offset | V.light_map_offset;
    return (a & 15) == 0 ? 16 : ((a & 3) == 0 ? 4 : 1);
}

// phase 3: the map cells of an env's record from its view rows, 8 bytes each {block, item + 1, lit, five mob
// classes} (:9241-9269).  A lane takes four cells of a row, bytes side by side.
__device__ __forceinline__ uint32_t span_word(const uint8_t* span, int dr, int o) {   // bytes o .. o + 3 of a row
    const uint32_t a = *reinterpret_cast<const uint32_t*>(span + row_byte(dr, o & ~3));
    const uint32_t b = *reinterpret_cast<const uint32_t*>(span + row_byte(dr, (o & ~3) + 4));
    return __funnelshift_r(a, b, 8 * (o & 3));
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {   // (__byte_perm drops the sign bit of a selector)
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
__device__ __forceinline__ uint32_t low_bytes(int k) { return k <= 0 ? 0u : (k >= 4 ? ~0u : (1u << 8 * k) - 1u); }
struct Cells { uint32_t w[4]; };   // first words of this lane's cells; the second ones hold mobs only
constexpr int kGroups = (kCols + 3) / 4;
static_assert(kRows * kGroups <= 32, "a lane a group");
__device__ __forceinline__ Cells make_cells(View v, int lane, const uint8_t* span) {
    const int dr = lane / kGroups, g = lane % kGroups, row = v.top() + dr, col = v.left() + 4 * g;
    Cells c = {{0u, 0u, 0u, 0u}};
    // (a level outside [0, 9) never comes out of the env; the reference would read outside
    // its maps there, here such an env gets unlit cells)
    if (dr >= kRows || (unsigned)row >= (unsigned)kMapSize || !v.level_ok()) return c;
    const int o = (v.left() & 15) + 4 * g;   // at most 23
    const uint32_t in = low_bytes(min(kMapSize - col, kCols - 4 * g)) & ~low_bytes(-col);
    const uint32_t lit = __vcmpgtu4(span_word(span, dr, o), kLit * 0x01010101u) & in;
    const uint32_t b = span_word(span + kSpan, dr, o) & lit, it = __vadd4(span_word(span + 2 * kSpan, dr, o), 0x01010101u) & lit;
    const uint32_t one = lit & 0x01010101u, lo = __byte_perm(b, it, 0x5140), hi = __byte_perm(b, it, 0x7362);
    c.w[0] = prmt(lo, one, 0xC410);   // {block, item, lit, 0}: selector 8 + i repeats the sign of byte i, here 0
    c.w[1] = prmt(lo, one, 0xD532);
    c.w[2] = prmt(hi, one, 0xE610);
    c.w[3] = prmt(hi, one, 0xF732);
    return c;
}
__device__ __forceinline__ void put_cells(const Cells& c, int lane, uint32_t* rec) {
    const int dr = lane / kGroups, g = lane % kGroups;
    if (dr >= kRows) return;
    uint32_t* d = rec + 2 * (dr * kCols + 4 * g);
#pragma unroll
    for (int i = 0; i < 4; i++)
        if (4 * g + i < kCols) { d[2 * i] = c.w[i]; d[2 * i + 1] = 0u; }
}
// a mob whose cell is lit, or 0 (the mobs of a level are those of the light plane that was copied), and its byte
__device__ __forceinline__ uint32_t lit_mob(View v, uint32_t pk, const uint8_t* span) {
    if (!(pk & 0x80000000u)) return 0u;
    const int cell = (pk >> 8) & 0xFFu;
    return span[row_byte(cell / kCols, (v.left() & 15) + cell % kCols)] > kLit ? pk : 0u;
}
__device__ __forceinline__ void put_mob(uint32_t pk, uint32_t* rec) {
    if (pk) reinterpret_cast<uint8_t*>(rec)[((pk >> 8) & 0xFFu) * 8 + ((pk >> 4) & 0xFu)] = (uint8_t)(pk & 0xFu);
}
__device__ __forceinline__ void store_record(uint8_t* records, int e, int lane, const uint32_t* rec) {
    uint32_t* dst = reinterpret_cast<uint32_t*>(records + (size_t)e * kRec);   // 4-byte aligned (996 = 4 x 249)
#pragma unroll
    for (int w = lane; w < kRecWords; w += 32) dst[w] = rec[w];
}

// Turns the view rows of a warp's kOwn envs in `span` into their records, in the same place; first: the first of the envs in the
// block, todo: those that there are
__device__ __forceinline__ uint32_t* assemble(const Gathered& S, const View (&v)[kOwn], uint32_t todo, int first, int lane, uint8_t* span) {
    Cells cells[kOwn];
    uint32_t mob[kOwn / 2];   // two envs at a time, 16 lanes each
#pragma unroll
    for (int k = 0; k < kOwn; k++) cells[k] = make_cells(v[k], lane, span + k * kPlanes * kSpan);
#pragma unroll
    for (int k = 0; k < kOwn; k += 2) {
        const int h = k + (lane >> 4);
        mob[k / 2] = 0u;
        if ((todo >> h & 1u) && (lane & 15) < kMobs)
            mob[k / 2] = lit_mob(lane < 16 ? v[k] : v[k + 1], S.mobs[first + h][lane & 15], span + h * kPlanes * kSpan);
    }
    __syncwarp();   // the rows are in registers
    uint32_t* rec = reinterpret_cast<uint32_t*>(span);   // [kOwn][kRecWords]
#pragma unroll
    for (int k = 0; k < kOwn; k++) {
        put_cells(cells[k], lane, rec + k * kRecWords);
        for (int j = lane; j < kTail; j += 32) rec[k * kRecWords + kMapWords + j] = __float_as_uint(S.tail[first + k][j]);
    }
    __syncwarp();   // the mob bytes land on cells other lanes have written
#pragma unroll
    for (int k = 0; k < kOwn; k += 2) put_mob(mob[k / 2], rec + (k + (lane >> 4)) * kRecWords);
    __syncwarp();
    return rec;
}

// (BYTES: the planes are not aligned to words.  A kernel of its own: beside the copies its loads made 1,024 envs 3 % slower.)
template <bool BYTES>
__global__ void __launch_bounds__(kBlockThreads, 4) k_record_rows(const __grid_constant__ Params P) {
    extern __shared__ __align__(16) uint8_t smem[];
    Shared& S = *reinterpret_cast<Shared*>(smem);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int e0 = blockIdx.x * kBlockEnvs, e = e0 + lane;
    const int n = P.v.num_envs, grain = copy_grain(P.v);
    wait_for_previous_kernel();
    bool live = e < P.n;
    int level = 0, top = 0, left = 0;
    if (live) {   // the flag and the position on their way together
        const uint8_t skipped = P.skip != nullptr ? ld_now(P.skip + e) : (uint8_t)0;
        level = soa(P.v.player_level, 0, n, e);
        top = soa(P.v.player_position, 0, n, e) - kRows / 2;
        left = soa(P.v.player_position, 1, n, e) - kCols / 2;
        live = skipped == 0;
    }
    const View mine = make_view(level, top, left);
    const CopyLane copy(lane);
    uint8_t* const span = S.span[warp];
    const uint32_t todo = __ballot_sync(0xffffffffu, live) >> (kOwn * warp) & ((1u << kOwn) - 1u);
    View v[kOwn];   // of this warp's envs, kOwn * warp + k of the block
#pragma unroll
    for (int k = 0; k < kOwn; k++) v[k].bits = __shfl_sync(0xffffffffu, mine.bits, kOwn * warp + k);
    Gather g;
    if (live) {
        g.load_fields(P.v, e, warp);
        g.load_of_level(P.v, e, warp, level);
    }
#pragma unroll
    for (int k = 0; k < kOwn; k++) {
        if (todo >> k & 1u) copy.start<BYTES>(P.v, e0 + kOwn * warp + k, v[k], grain, span + k * kPlanes * kSpan);
    }
    if (live) g.finish(P.v, e, lane, warp, level, top, left, S);
    wait_spans();
    __syncthreads();
    const uint32_t* rec = assemble(S, v, todo, kOwn * warp, lane, span);
    if (todo == (1u << kOwn) - 1u && (reinterpret_cast<uintptr_t>(P.records) & 15) == 0) {
        // the warp's records in one bulk copy
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(P.records + (size_t)(e0 + kOwn * warp) * kRec),
                         "r"((uint32_t)__cvta_generic_to_shared(rec)), "r"(kOwn * kRec) : "memory");
            asm volatile("cp.async.bulk.commit_group;\n\tcp.async.bulk.wait_group.read 0;" ::: "memory");
        }
    } else {
        for (int k = 0; k < kOwn; k++)
            if (todo >> k & 1u) store_record(P.records, e0 + kOwn * warp + k, lane, rec + k * kRecWords);
    }
}

// ------------------------------------------------------------------ list of envs
// The envs named by a device-side list (first int32 of every entry): a few that are being reset, anywhere in
// the batch, so what counts is the chain of dependent loads and not coalescing.  A warp takes an
// env: entry -> every scalar, the level and the position, all lanes at once -> mobs and map rows -> record.  About 250
// entries of 65,536 envs: 26 us with a block for 32 entries, now 4 (9.8 from cold caches).  A long list is another
// matter: there a block takes 32 entries at a time as k_record_rows does, see list_block.
// The fields of the tail by position: which field pointer of the view, which element, how it is scaled.
enum Scale : uint8_t { S_SQRT10, S_10, S_2, S_4, S_INT, S_F10, S_FLOAT, S_FLAG, S_DIR, S_KILLED, S_BOSS };
struct TailField { uint8_t field, elem, scale; };
#define CFX_FIELD(name) (uint8_t)((offsetof(cfx_env_view, name) - offsetof(cfx_env_view, player_position)) / sizeof(void*))
// the 51 scalars in the order of craftax_encode_scalar_observation_tail_at (:2429-2487)
__device__ const TailField kTailFields[kTail] = {
    {CFX_FIELD(inv_wood), 0, S_SQRT10}, {CFX_FIELD(inv_stone), 0, S_SQRT10}, {CFX_FIELD(inv_coal), 0, S_SQRT10},
    {CFX_FIELD(inv_iron), 0, S_SQRT10}, {CFX_FIELD(inv_diamond), 0, S_SQRT10}, {CFX_FIELD(inv_sapphire), 0, S_SQRT10},
    {CFX_FIELD(inv_ruby), 0, S_SQRT10}, {CFX_FIELD(inv_sapling), 0, S_SQRT10}, {CFX_FIELD(inv_torches), 0, S_SQRT10},
    {CFX_FIELD(inv_arrows), 0, S_SQRT10}, {CFX_FIELD(inv_books), 0, S_2}, {CFX_FIELD(inv_pickaxe), 0, S_4},
    {CFX_FIELD(inv_sword), 0, S_4}, {CFX_FIELD(sword_enchantment), 0, S_INT}, {CFX_FIELD(bow_enchantment), 0, S_INT},
    {CFX_FIELD(inv_bow), 0, S_INT}, {CFX_FIELD(inv_potions), 0, S_SQRT10}, {CFX_FIELD(inv_potions), 1, S_SQRT10},
    {CFX_FIELD(inv_potions), 2, S_SQRT10}, {CFX_FIELD(inv_potions), 3, S_SQRT10}, {CFX_FIELD(inv_potions), 4, S_SQRT10},
    {CFX_FIELD(inv_potions), 5, S_SQRT10}, {CFX_FIELD(player_health), 0, S_F10}, {CFX_FIELD(player_food), 0, S_10},
    {CFX_FIELD(player_drink), 0, S_10}, {CFX_FIELD(player_energy), 0, S_10}, {CFX_FIELD(player_mana), 0, S_10},
    {CFX_FIELD(player_xp), 0, S_10}, {CFX_FIELD(player_dexterity), 0, S_10}, {CFX_FIELD(player_strength), 0, S_10},
    {CFX_FIELD(player_intelligence), 0, S_10}, {CFX_FIELD(player_direction), 1, S_DIR}, {CFX_FIELD(player_direction), 2, S_DIR},
    {CFX_FIELD(player_direction), 3, S_DIR}, {CFX_FIELD(player_direction), 4, S_DIR}, {CFX_FIELD(inv_armour), 0, S_2},
    {CFX_FIELD(inv_armour), 1, S_2}, {CFX_FIELD(inv_armour), 2, S_2}, {CFX_FIELD(inv_armour), 3, S_2},
    {CFX_FIELD(armour_enchantments), 0, S_INT}, {CFX_FIELD(armour_enchantments), 1, S_INT},
    {CFX_FIELD(armour_enchantments), 2, S_INT}, {CFX_FIELD(armour_enchantments), 3, S_INT},
    {CFX_FIELD(light_level), 0, S_FLOAT}, {CFX_FIELD(is_sleeping), 0, S_FLAG}, {CFX_FIELD(is_resting), 0, S_FLAG},
    {CFX_FIELD(learned_spells), 0, S_FLAG}, {CFX_FIELD(learned_spells), 1, S_FLAG}, {CFX_FIELD(player_level), 0, S_10},
    {CFX_FIELD(monsters_killed), 0, S_KILLED}, {CFX_FIELD(boss_timesteps_to_spawn_this_round), 0, S_BOSS}};

// the raw bits of tail scalar f (S_KILLED is read by its own lane later, when the level is known)
__device__ __forceinline__ uint32_t tail_raw(const cfx_env_view& V, const TailField& f, int e) {
    const void* base = (&reinterpret_cast<const void* const&>(V.player_position))[f.field];
    const size_t elem = f.scale == S_DIR ? 0 : f.elem, i = elem * (size_t)V.num_envs + (size_t)e;
    if (f.scale == S_KILLED) return 0u;
    return f.scale == S_FLAG ? (uint32_t)ld_now(reinterpret_cast<const uint8_t*>(base) + i) : ld_now(reinterpret_cast<const uint32_t*>(base) + i);
}
__device__ __forceinline__ float tail_value(const TailField& f, uint32_t raw, bool killed, bool mob_alive) {
    const float v = (float)(int32_t)raw;
    switch (f.scale) {
        case S_SQRT10: return sqrtf(v) * (1.0f / 10.0f);
        case S_10: return v * (1.0f / 10.0f);
        case S_2: return v * (1.0f / 2.0f);
        case S_4: return v * (1.0f / 4.0f);
        case S_INT: return v;
        case S_F10: return __uint_as_float(raw) * (1.0f / 10.0f);
        case S_FLOAT: return __uint_as_float(raw);
        case S_FLAG: return raw != 0 ? 1.0f : 0.0f;
        case S_DIR: return (int32_t)raw == f.elem ? 1.0f : 0.0f;
        case S_KILLED: return killed ? 1.0f : 0.0f;
        default: return !mob_alive && (int32_t)raw <= 0 ? 1.0f : 0.0f;
    }
}

struct ListShared {
    uint32_t rec[kRecWords + 3];
    __align__(16) uint8_t span[kPlanes * kSpan];
};
static_assert(sizeof(ListShared) % 16 == 0, "alignment");
constexpr int kListThreads = 128, kListWarps = kListThreads / 32;
struct ListBlock : Gathered {
    __align__(16) uint8_t span[kListWarps][kOwn * kPlanes * kSpan];
};
union ListMemory {
    ListShared warp[kListWarps];
    ListBlock block;
};
static_assert(sizeof(ListMemory) <= 48 * 1024, "static shared memory");
// Lists of more entries than this for each warp of the grid go by blocks.  65,536 envs, 2,368 warps, envs chosen at random, three sets of buffers, us by warps /
// by blocks: 250 entries 4.1 / 8.0, 2,368 5.8 / 9.7, 4,736 11.8 / 11.8, 7,104 17.1 / 13.9, 16,384 33.4 / 18.6, all of them 119 / 52.
constexpr int kListPerWarp = 2;

// 32 entries of the list from `base` on, lane = entry in the loads of the fields, a warp four envs at a time in the rest
template <bool BYTES>
__device__ __forceinline__ void list_block(const Params& P, ListBlock& S, const CopyLane& copy, int grain, int base, int count) {
    const cfx_env_view& V = P.v;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = V.num_envs;
    int e = -1, level = 0, top = 0, left = 0;
    if (base + lane < count) e = *reinterpret_cast<const int32_t*>(P.list + (size_t)(base + lane) * P.list_stride);
    const bool live = e >= 0 && e < n;
    if (live) {
        level = soa(V.player_level, 0, n, e);
        top = soa(V.player_position, 0, n, e) - kRows / 2;
        left = soa(V.player_position, 1, n, e) - kCols / 2;
    }
    const View mine = make_view(level, top, left);
    const uint32_t all = __ballot_sync(0xffffffffu, live);
    uint8_t* const span = S.span[warp];
    View v[kOwn];
    auto copies = [&](int first) {
#pragma unroll
        for (int k = 0; k < kOwn; k++) {
            v[k].bits = __shfl_sync(0xffffffffu, mine.bits, first + k);
            const int env = __shfl_sync(0xffffffffu, e, first + k);
            if (all >> (first + k) & 1u) copy.start<BYTES>(V, env, v[k], grain, span + k * kPlanes * kSpan);
        }
    };
    constexpr int kWarpEnvs = kBlockEnvs / kListWarps;
    copies(kWarpEnvs * warp);
#pragma unroll 1
    for (int part = warp; part < kWarps; part += kListWarps)
        if (live) {
            Gather g;
            g.load_fields(V, e, part);
            g.load_of_level(V, e, part, level);
            g.finish(V, e, lane, part, level, top, left, S);
        }
    wait_spans();
    __syncthreads();
#pragma unroll 1
    for (int i = 0; i < kWarpEnvs; i += kOwn) {
        const int first = kWarpEnvs * warp + i;
        if (i > 0) {
            copies(first);
            wait_spans();
        }
        const uint32_t todo = all >> first & ((1u << kOwn) - 1u);
        const uint32_t* rec = assemble(S, v, todo, first, lane, span);
        for (int k = 0; k < kOwn; k++) {
            const int env = __shfl_sync(0xffffffffu, e, first + k);
            if (todo >> k & 1u) store_record(P.records, env, lane, rec + k * kRecWords);
        }
        __syncwarp();
    }
    __syncthreads();
}

template <bool BYTES>
__global__ void __launch_bounds__(kListThreads, 4) k_record_rows_list(const __grid_constant__ Params P) {
    __shared__ ListMemory M;
    const cfx_env_view& V = P.v;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = V.num_envs, grain = copy_grain(V);
    ListShared& S = M.warp[warp];
    const CopyLane copy(lane);
    const TailField f0 = kTailFields[lane], f1 = kTailFields[min(lane + 32, kTail - 1)];
    wait_for_previous_kernel();
    const int count = *P.count_dev;
    const int stride = (int)gridDim.x * kListWarps;
    if (count > kListPerWarp * stride) {
        for (int base = (int)blockIdx.x * kBlockEnvs; base < count; base += (int)gridDim.x * kBlockEnvs)
            list_block<BYTES>(P, M.block, copy, grain, base, count);
        return;
    }
    for (int i = (int)blockIdx.x * kListWarps + warp; i < count; i += stride) {
        const int e = *reinterpret_cast<const int32_t*>(P.list + (size_t)i * P.list_stride);
        if (e < 0 || e >= n) continue;
        const int level = soa(V.player_level, 0, n, e);
        const int top = soa(V.player_position, 0, n, e) - kRows / 2, left = soa(V.player_position, 1, n, e) - kCols / 2;
        const uint32_t raw0 = tail_raw(V, f0, e), raw1 = lane + 32 < kTail ? tail_raw(V, f1, e) : 0u;
        const View v = make_view(level, top, left);
        copy.start<BYTES>(V, e, v, grain, S.span);
        const bool killed = (unsigned)level < (unsigned)kLevels && soa(V.monsters_killed, level, n, e) >= kKilledToClear;
        // lane 3 c + i: slot i of mob class c
        const int c = lane / kSlots, slot = lane % kSlots;
        uint32_t pk = 0;
        bool mask = false;
        if (lane < kMobs && slot < (c == 2 ? 2 : 3)) {
            const int idx = mob_index(c, jax_index(level, kLevels), slot);
            mask = soa(V.mob_mask, idx, n, e) != 0;
            pk = pack_mob(c, soa(V.mob_type_id, idx, n, e), mask, soa(V.mob_position, idx * 2, n, e),
                          soa(V.mob_position, idx * 2 + 1, n, e), top, left);
        }
        const bool alive = __any_sync(0xffffffffu, mask && (c == 0 || c == 2));
        const uint32_t next1 = __shfl_down_sync(0xffffffffu, pk, 1), next2 = __shfl_down_sync(0xffffffffu, pk, 2);
        if ((slot < 2 && same_cell(pk, next1)) || (slot < 1 && same_cell(pk, next2))) pk = 0;   // a later slot covers it
        float* tail = reinterpret_cast<float*>(S.rec + kMapWords);
        tail[lane] = tail_value(f0, raw0, killed, alive);
        if (lane + 32 < kTail) tail[lane + 32] = tail_value(f1, raw1, killed, alive);
        wait_spans();
        put_cells(make_cells(v, lane, S.span), lane, S.rec);
        __syncwarp();
        put_mob(lit_mob(v, pk, S.span), S.rec);
        __syncwarp();
        store_record(P.records, e, lane, S.rec);
        __syncwarp();
    }
}

static int make_params(const char* who, const cfx_env_view* view, uint8_t* records, Params* P) {
    CFX_REQUIRE(view != nullptr && records != nullptr, "%s: bad argument", who);
    CFX_REQUIRE(view->num_envs > 0 && view->state_base != nullptr && view->state_stride > 0,
                "%s: the view has no envs or no state block", who);
    CFX_REQUIRE(((uintptr_t)records & 3) == 0, "%s: records must be 4-byte aligned", who);
    // every field pointer of the view sits between player_position and mob_type_id
    const void* const* first = reinterpret_cast<const void* const*>(&view->player_position);
    const void* const* last = reinterpret_cast<const void* const*>(&view->mob_type_id);
    for (const void* const* q = first; q <= last; q++)
        CFX_REQUIRE(*q != nullptr, "%s: field pointer %d of the view is NULL", who, (int)(q - first));
    P->v = *view;
    P->records = records;
    P->skip = nullptr; P->list = nullptr; P->list_stride = 0; P->count_dev = nullptr;
    P->n = view->num_envs;
    return CFX_OK;
}

static_assert(4 * (sizeof(Shared) + 1024) <= 228 * 1024, "four blocks an SM");
static_assert(offsetof(cfx_env_view, mob_type_id) - offsetof(cfx_env_view, player_position) == 39 * sizeof(void*),
              "the field pointers of cfx_env_view are contiguous (make_params walks them)");


// ------------------------------------------------------------------ classic game
// record_obs_kernel (craftax_classic.cu:1884-1890) gives every env a thread that writes its 148
// bytes one by one: 148 store instructions per warp, each touching 32 different records.  Here a
// block gathers the records of 64 consecutive envs, thread per env (the SoA loads of a warp are
// contiguous, and all in flight at once), puts them together word by word in registers, and writes the 9,472
// contiguous bytes out of shared memory as coalesced 16-byte words (row length 37 words: no bank conflicts).
// The seven map rows of a view are 224 contiguous bytes: the warp copies those of two envs an
// instruction to shared memory (whole rows: what is read from memory is 32-byte sectors anyway), where a
// thread then takes the nine nibbles of a row from two words.  Loads of these words from the map
// itself, 14 a thread, touch 32 cache lines an instruction: 20 of 41 us of a cache's time.  262,144 envs: a load per cell
// 103 us, words from the map 41.5, rows through shared memory 27.3 (102 MB read from DRAM, 39 MB written), with 64 bytes a miss 25.7
// (86 MB); 65,536 envs 12.4 -> 8.2 us.
constexpr int kClRows = 7, kClCols = 9, kClCells = kClRows * kClCols, kClMap = 64, kClRowBytes = 32;
constexpr int kClSpan = kClRows * kClRowBytes + 16;   // 60 words: as few bank conflicts as 16-byte pieces allow
constexpr int kClInv = 12, kClOutOfBounds = 1, kClBlockEnvs = 64, kClWords = kClassicRec / 4;
static_assert(2 * kClCells + kClInv + 6 + 4 == kClassicRec && kClassicRec % 4 == 0, "classic record layout");

// bytes of a record put together in order, word by word; positions are compile-time constants once unrolled
struct ClassicWords {
    uint32_t w[kClWords];
    __device__ __forceinline__ void put(int pos, uint32_t v, int bytes) {   // v < 2^(8 bytes)
        w[pos / 4] |= v << (8 * (pos % 4));
        if (pos % 4 + bytes > 4) w[pos / 4 + 1] |= v >> (32 - 8 * (pos % 4));
    }
};

__global__ void __launch_bounds__(kClBlockEnvs) k_classic_record_rows(const __grid_constant__ cfx_classic_env_view V,
                                                                     uint8_t* __restrict__ records, int n_envs) {
    // the envs' map rows (the word before the first and the one after the last are read, and masked), then the records
    __shared__ __align__(16) uint8_t smem[16 + kClBlockEnvs * kClSpan + 16];
    static_assert(sizeof(smem) >= kClBlockEnvs * kClassicRec, "the records lie where the rows were");
    const int t = threadIdx.x, lane = t & 31;
    const int e0 = blockIdx.x * kClBlockEnvs, e = min(e0 + t, n_envs - 1);
    const int n = V.num_envs;
    wait_for_previous_kernel();
    const int pr = soa(V.player_r, 0, n, e), pc = soa(V.player_c, 0, n, e);
    int8_t inv[kClInv];
#pragma unroll
    for (int i = 0; i < kClInv; i++) inv[i] = soa(V.inv, i, n, e);
    const int8_t intr[5] = {soa(V.health, 0, n, e), soa(V.food, 0, n, e), soa(V.drink, 0, n, e), soa(V.energy, 0, n, e),
                            soa(V.player_dir, 0, n, e)};
    const uint8_t sleeping = soa(V.is_sleeping, 0, n, e);
    const float light = soa(V.light_level, 0, n, e);
    constexpr int kMobsCl = 11;
    const int16_t* const mob_r[4] = {V.zombie_r, V.cow_r, V.skel_r, V.arrow_r};
    const int16_t* const mob_c[4] = {V.zombie_c, V.cow_c, V.skel_c, V.arrow_c};
    const uint8_t* const mob_m[4] = {V.zombie_mask, V.cow_mask, V.skel_mask, V.arrow_mask};
    constexpr int kKind[kMobsCl] = {0, 0, 0, 1, 1, 1, 2, 2, 3, 3, 3}, kSlot[kMobsCl] = {0, 1, 2, 0, 1, 2, 0, 1, 0, 1, 2};
    int16_t mr[kMobsCl], mc[kMobsCl];
    uint8_t on[kMobsCl];
#pragma unroll
    for (int i = 0; i < kMobsCl; i++) {
        on[i] = soa(mob_m[kKind[i]], kSlot[i], n, e);
        mr[i] = soa(mob_r[kKind[i]], kSlot[i], n, e);
        mc[i] = soa(mob_c[kKind[i]], kSlot[i], n, e);
    }
    // view rows: blocks (a nibble per map column; 1 outside the map)  (:1061-1100)
    // first byte and word of the view's columns in a map row (a view that is off the map is masked as a whole)
    const int o = (pc - 4) >> 1, wi = min(max(o >> 2, -1), kClRowBytes / 4 - 1);
    uint8_t* const span = smem + 16 + t * kClSpan;
    const uintptr_t align = reinterpret_cast<uintptr_t>(V.map_packed) | V.map_stride;
    if ((align & 15) == 0) {
        const int j = lane & 15, half = lane >> 4;
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
            const int row = __shfl_sync(0xffffffffu, pr, i + half) - 3 + (j >> 1), env = __shfl_sync(0xffffffffu, e, i + half);
            if (j < 2 * kClRows && row >= 0 && row < kClMap) {
                const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem + 16 + ((t & ~31) + i + half) * kClSpan + 16 * j);
                const uint8_t* q = V.map_packed + (size_t)env * V.map_stride + row * kClRowBytes + 16 * (j & 1);
                asm volatile("cp.async.cg.shared.global.L2::64B [%0], [%1], 16;" ::"r"(d), "l"(q) : "memory");
            }
        }
    } else {
        const uint8_t* map = V.map_packed + (size_t)e * V.map_stride;
        for (int k = 0; k < 2 * kClRows; k++) {
            const int row = pr - 3 + k / 2, i = wi + k % 2;
            if (row < 0 || row >= kClMap || i < 0 || i >= kClRowBytes / 4) continue;
            const uint8_t* q = map + row * kClRowBytes + 4 * i;
            uint32_t w;
            if ((align & 3) == 0) w = ld_now(reinterpret_cast<const uint32_t*>(q));
            else w = ld_now(q) | (uint32_t)ld_now(q + 1) << 8 | (uint32_t)ld_now(q + 2) << 16 | (uint32_t)ld_now(q + 3) << 24;
            *reinterpret_cast<uint32_t*>(span + k / 2 * kClRowBytes + 4 * i) = w;
        }
    }
    ClassicWords R;
#pragma unroll
    for (int i = 0; i < kClWords; i++) R.w[i] = 0u;
    // inventory, intrinsics, direction, sleeping, light  (:1590-1603)
    constexpr int kTailPos = 2 * kClCells;
#pragma unroll
    for (int i = 0; i < kClInv; i++) R.put(kTailPos + i, (uint8_t)inv[i], 1);
#pragma unroll
    for (int i = 0; i < 5; i++) R.put(kTailPos + kClInv + i, (uint8_t)intr[i], 1);
    R.put(kTailPos + kClInv + 5, sleeping ? 1u : 0u, 1);
    R.put(kTailPos + kClInv + 6, __float_as_uint(light), 4);
    // columns of the view that lie on the map, a nibble each
    uint64_t in = 0;
#pragma unroll
    for (int c = 0; c < kClCols; c++)
        if (pc - 4 + c >= 0 && pc - 4 + c < kClMap) in |= 15ull << (4 * c);
    const int shift = 8 * (o & 3) + 4 * (pc & 1);
    wait_spans();
#pragma unroll
    for (int r = 0; r < kClRows; r++) {
        const bool row_in = pr - 3 + r >= 0 && pr - 3 + r < kClMap;
        const uint64_t keep = row_in ? in : 0ull;
        const uint32_t* w = reinterpret_cast<const uint32_t*>(span + r * kClRowBytes) + wi;
        const uint64_t v = (((uint64_t)w[1] << 32 | w[0]) >> shift & keep) | (0x111111111ull * kClOutOfBounds & ~keep);
        const uint32_t lo = (uint32_t)v, even = lo & 0x0F0F0F0Fu, odd = lo >> 4 & 0x0F0F0F0Fu;
        R.put(r * kClCols, __byte_perm(even, odd, 0x5140), 4);
        R.put(r * kClCols + 4, __byte_perm(even, odd, 0x7362), 4);
        R.put(r * kClCols + 8, (uint32_t)(v >> 32) & 15u, 1);
    }
    __syncthreads();   // the rows of all warps are in registers
    uint32_t* const srec = reinterpret_cast<uint32_t*>(smem);
#pragma unroll
    for (int i = 0; i < kClWords; i++) srec[t * kClWords + i] = R.w[i];
    // mobs inside the view set their bit  (:1102-1125)
    uint8_t* mobs = reinterpret_cast<uint8_t*>(srec + t * kClWords) + kClCells;
#pragma unroll
    for (int i = 0; i < kMobsCl; i++) {
        const int dr = mr[i] - pr + 3, dc = mc[i] - pc + 4;
        if (on[i] != 0 && (unsigned)dr < (unsigned)kClRows && (unsigned)dc < (unsigned)kClCols)
            mobs[dr * kClCols + dc] |= (uint8_t)(1 << kKind[i]);
    }
    __syncthreads();
    // the block's records are contiguous in global memory: 37 words per env
    const int words = min(kClBlockEnvs, n_envs - e0) * kClWords;
    uint32_t* dst = reinterpret_cast<uint32_t*>(records + (size_t)e0 * kClassicRec);
    const int quads = (reinterpret_cast<uintptr_t>(records) & 15) == 0 ? words / 4 : 0;
    for (int q = t; q < quads; q += kClBlockEnvs)
        reinterpret_cast<uint4*>(dst)[q] = reinterpret_cast<const uint4*>(srec)[q];
    for (int w = 4 * quads + t; w < words; w += kClBlockEnvs) dst[w] = srec[w];
}

}  // namespace record
}  // namespace cfx

using namespace cfx;

extern "C" int cfx_record_obs(int device, const cfx_env_view* view, uint8_t* records, int n, const uint8_t* skip,
                              void* stream) {
    record::Params P;
    int rc = record::make_params("cfx_record_obs", view, records, &P);
    if (rc != CFX_OK) return rc;
    CFX_REQUIRE(n > 0 && n <= view->num_envs, "cfx_record_obs: n=%d outside (0, num_envs=%d]", n, view->num_envs);
    CFX_GUARD(device);
    P.n = n;
    P.skip = skip;
    const unsigned blocks = (unsigned)((n + record::kBlockEnvs - 1) / record::kBlockEnvs);
    auto launch = [&](auto bytes) {
        constexpr auto kernel = record::k_record_rows<decltype(bytes)::value>;
        const int rc = allow_smem<kernel, (int)sizeof(record::Shared)>();
        if (rc) return rc;
        return launch_chained(kernel, dim3(blocks), record::kBlockThreads, sizeof(record::Shared), (cudaStream_t)stream, P);
    };
    return record::copy_grain(*view) == 1 ? launch(std::true_type()) : launch(std::false_type());
}

extern "C" int cfx_record_obs_list(int device, const cfx_env_view* view, uint8_t* records, const void* list,
                                   int list_stride, const int* count_dev, void* stream) {
    record::Params P;
    int rc = record::make_params("cfx_record_obs_list", view, records, &P);
    if (rc != CFX_OK) return rc;
    CFX_REQUIRE(list != nullptr && count_dev != nullptr && list_stride >= 4 && list_stride % 4 == 0,
                "cfx_record_obs_list: bad list");
    CFX_GUARD(device);
    P.list = (const uint8_t*)list;
    P.list_stride = list_stride;
    P.count_dev = count_dev;
    // the count is on the device: a fixed grid of at most four blocks an SM walks the list, a warp an entry
    // (the reference uses at most 128 blocks of 8 warps for its list pass, :11941)
    int blocks = (view->num_envs + record::kListWarps - 1) / record::kListWarps;
    if (blocks > 592) blocks = 592;
    return launch_chained(record::copy_grain(*view) == 1 ? record::k_record_rows_list<true> : record::k_record_rows_list<false>,
                          dim3((unsigned)blocks), record::kListThreads, 0, (cudaStream_t)stream, P);
}

extern "C" int cfx_classic_record_obs(int device, const cfx_classic_env_view* view, uint8_t* records, int n,
                                      void* stream) {
    CFX_REQUIRE(view != nullptr && records != nullptr, "cfx_classic_record_obs: bad argument");
    CFX_REQUIRE(view->num_envs > 0 && n > 0 && n <= view->num_envs,
                "cfx_classic_record_obs: n=%d outside (0, num_envs=%d]", n, view->num_envs);
    CFX_REQUIRE(((uintptr_t)records & 3) == 0, "cfx_classic_record_obs: records must be 4-byte aligned");
    CFX_REQUIRE(view->map_packed != nullptr && view->map_stride >= 64 * 32,
                "cfx_classic_record_obs: the view has no packed map");
    // every field pointer of the view sits between player_r and light_level
    const void* const* first = reinterpret_cast<const void* const*>(&view->player_r);
    const void* const* last = reinterpret_cast<const void* const*>(&view->light_level);
    for (const void* const* q = first; q <= last; q++)
        CFX_REQUIRE(*q != nullptr, "cfx_classic_record_obs: field pointer %d of the view is NULL", (int)(q - first));
    CFX_GUARD(device);
    const unsigned blocks = (unsigned)((n + record::kClBlockEnvs - 1) / record::kClBlockEnvs);
    return launch_chained(record::k_classic_record_rows, dim3(blocks), record::kClBlockEnvs, 0, (cudaStream_t)stream, *view, records, n);
}
