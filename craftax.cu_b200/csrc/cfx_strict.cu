// Strict-fp32 forward on CUDA cores (precision CFX_PREC_FP32) plus the
// stand-alone expand / sampler / uniform stages.
//
// Every dot product is accumulated with fmaf in ascending input order, which
// is the order of the reference's scalar policy kernel (k_policy_ref_l3,
// craftax_full.cu:9778-9854); this file is compiled with -fmad=false like the
// reference's full-game build (Makefile:27), so the cell arithmetic rounds at
// the same places.  It is the high-accuracy mode of the library and the
// on-device yardstick for the tensor-core kernel at sizes a CPU cannot check.
#include <cuda_bf16.h>

#include <atomic>
#include <type_traits>

#include "cfx_common.cuh"
#include "cfx_f32x2.cuh"
#include "cfx_sampler.cuh"
#include "cfx_strict.h"

namespace cfx {

constexpr int kSMs = 148;

// ---------------------------------------------------------------- expand
// features[e][f] = (float)rec[e][f] for f < 792, raw fp32 bits for the tail
// (k_expand_obs, craftax_full.cu:10028-10053).  One thread per output element;
// consecutive threads write consecutive floats.
__global__ void k_expand(const uint8_t* __restrict__ rec, float* __restrict__ out, int n) {
    size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)n * kObs) return;
    int f = (int)(idx % kObs);
    size_t e = idx / kObs;
    const uint8_t* r = rec + e * kRec;
    float x;
    if (f < kMap) {
        x = (float)r[f];
    } else {
        // records are 4-byte aligned (996 = 4 * 249, 792 = 4 * 198)
        x = *reinterpret_cast<const float*>(r + kMap + 4 * (f - kMap));
    }
    out[idx] = x;
}

// ---------------------------------------------------------------- tiling of the fp32 layers
// The encoder and the MinGRU layers are fp32 matrix products whose sums run in ascending input
// order, so nothing may be split along the inputs; the work is split over (env, unit) tiles.  They
// are bound by the FMA pipe (128 lanes per clock and SM), and a thread that loads an operand for few FMAs by
// shared-memory reads instead (a cycle per operand register and warp, broadcast or not).  In a layer a lane
// owns TM envs x 4 units, all three gates, a warp 4 TM envs x 32 units (lane = 8 groups of units x 4
// groups of envs), and a block is WM x WU such warps.  Activations travel between the kernels in tiles of
// 32 envs, [n / 32][H][32], and the gate matrices in tiles of 64 (32) units, so that both operands of a k step are
// contiguous in shared memory; two units at a time go through the packed FMA (`fma.rn.f32x2`, the rounding of fmaf), which leaves
// issue slots for the operand reads.  (One env and unit at a time: 199 us against 147 at 4,096 envs, hidden 256, depth 2.  Pairs of envs
// times pairs of units, straight and crossed, which need half as many register moves: 157.)
// (The doubled input of a pair is made with register moves: stored doubled it costs 8 more operand
// registers from shared memory a k step, and the layer kernel went from 52 to 59 us at 4,096 envs.  From tensor memory, as it is or
// doubled, a loop of nothing but the sums of a layer keeps the FMA pipe 88 and 78 % busy, from shared memory 89 %.)
// The TM envs of a lane among the 4 TM of its warp: quads of the 16 envs that the four groups g of lanes have together, then
// a pair of 8, then one of 4, so that a lane's envs are aligned words in shared memory for any TM.
template <int TM> struct Envs {
    static constexpr int kQuads = TM / 4, kPair = TM % 4 / 2, kOne = TM % 2, kParts = kQuads + kPair + kOne;
    static __host__ __device__ constexpr int first(int part) { return part < kQuads ? 4 * part : 4 * kQuads + (part > kQuads ? 2 * kPair : 0); }
    static __host__ __device__ constexpr int count(int part) { return part < kQuads ? 4 : (part == kQuads && kPair ? 2 : 1); }
    static __device__ __forceinline__ int at(int part, int g) { return 4 * first(part) + count(part) * g; }   // first env of a part
};
// its inputs, each doubled for the packed FMA; x: those of the warp's first env
template <int TM> struct Frag {
    uint64_t v[TM];
    __device__ __forceinline__ void load(const float* x, int g) {
        using E = Envs<TM>;
#pragma unroll
        for (int p = 0; p < E::kParts; p++) {
            const float* q = x + E::at(p, g);
            uint64_t* d = v + E::first(p);
            if (E::count(p) == 4) {
                const float4 f = *reinterpret_cast<const float4*>(q);
                d[0] = f2pack(f.x, f.x); d[1] = f2pack(f.y, f.y); d[2] = f2pack(f.z, f.z); d[3] = f2pack(f.w, f.w);
            } else if (E::count(p) == 2) {
                const float2 f = *reinterpret_cast<const float2*>(q);
                d[0] = f2pack(f.x, f.x); d[1] = f2pack(f.y, f.y);
            } else {
                d[0] = f2pack(q[0], q[0]);
            }
        }
    }
};
// Loads that are issued where they stand, and see what a kernel in front has written
__device__ __forceinline__ uint32_t ld_now(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void ld_now4(const float* p, float* v) {
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p));
}
// N envs side by side of a unit
template <int N> __device__ __forceinline__ void store_envs(float* p, const float (&v)[4]) {
    if constexpr (N == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else if constexpr (N == 2) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
    else *p = v[0];
}
__device__ __forceinline__ void store_envs(float* p, const float (&v)[4], int count) {   // (count is a constant once unrolled)
    if (count == 4) store_envs<4>(p, v);
    else if (count == 2) store_envs<2>(p, v);
    else store_envs<1>(p, v);
}
// 16 bytes global -> shared in flight (zeros where `on` is false); a source that is only 4-byte
// aligned goes as four words
__device__ __forceinline__ void copy16(float* dst, const float* src, bool on, bool aligned) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if (aligned) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(on ? 16 : 0) : "memory");
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + 4 * i), "l"(src + i), "r"(on ? 4 : 0) : "memory");
    }
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// `early` of the kernels: start the next kernel at once; the weights may be read before the kernel in front has
// ended (those of a handle are only ever written by calls that wait for the device)
constexpr int kLaunchNext = 1, kWeightsReady = 2;

// element (unit k, env e) of the activations
__host__ __device__ __forceinline__ size_t act_at(size_t e, int k, int H) { return ((e >> 5) * (size_t)H + (size_t)k) * 32 + (e & 31); }

// ---------------------------------------------------------------- encoder
// h_enc[k][e] = b_enc[k] + sum_f x[e][f] * W_enc[f][k], ascending f.  A lane owns TM envs x G groups of 4
// units, the groups 32 units apart.  Few warps of such tiles fall to an SM scheduler (one at 4,096 envs,
// hidden 256), so everything but the sums is taken out of them: four warps of a block fill the stages (record bytes ->
// fp32; W_enc rows by asynchronous copies), four multiply, and named barriers hand the stages over.
// A feature that is zero in all envs of a block is left out: its products change no sum (but the sign of one that is still -0).  Most bytes of a
// record are zero, five of a cell's eight unless there is a mob: of the 843 features 410 are left in blocks of 56 envs of a game, 546 with a mob of each
// class on every hundredth cell.  Zero times a weight that is infinite or not a number is not zero: with such weights (odd_weights, looked for when the
// weights are laid out) nothing is left out.  The block copies its records' maps to shared memory, ORs them over the envs on their way, and makes a list of
// the features that are left, from which the stages are filled.  What the list and the map give for a stage is loaded before it is used: row by row the latencies
// of shared memory add up.  Narrow tiles fill several rows an instruction; where nothing is left out a word of the map gives four features.  Stages of 32 rows:
// with 16 the barriers cost 2 to 6 %.
// Bound by the FMA pipe, the operands' reads of shared memory beside it, and some 3,000 cycles until the first stage is there.  us a forward with every feature,
// without a list; now; and now with records that have no zeros, which no game writes.  Hidden 256, depth 2: 32 envs 32.7, 29.7, 33.6, 128 43.6, 37.6, 43.1, 1,024
// 58.8, 55.5, 60.0, 2,048 84.4, 73.4, 83.8, 4,096 123.5, 111.7, 122.1; depth 1: 65,536 1,075, 911, 1,059; 4,096, hidden 128 53.3, 42.5, 52.8; 8,192, hidden
// 512, depth 3 828, 780, 821.
constexpr int kEncWarps = 8, kEncFill = 4;   // warps of a block, those of them that fill the stages
constexpr int kMapRounds = (kMap / 4 + 31) / 32, kMapPitch = kMap + 4;   // rounds of a warp's lanes with a word of a record each; bytes from one env's map to the next's
constexpr int kMapGroups = (kMap + 31) / 32, kGroups = kMapGroups + (kTail + 31) / 32;   // features by 32
static_assert(kGroups < 32 && 4 * kMapRounds < 32 && kMap % 4 == 0 && kMapPitch % 8 == 4, "a lane a group; a lane an env without bank conflicts");
template <int TM, int G, int WU, int UL> struct Enc {   // WU of the four warps side by side along the units, UL units of a group a lane
    static constexpr int WM = 4 / WU, BM = UL * TM * WM, BU = 32 * G * WU;   // envs, units
    static constexpr int XS = BM + (BM % 8 == 0 ? 4 : 0);               // row stride of x
    static constexpr int K = 32, S = TM == 1 ? 6 : G == 1 ? 4 : WU == 2 && TM <= 6 ? 3 : 2, R = S * K;   // rows of a stage, stages
    static constexpr int kOffMap = R * (XS + BU) * 4, kOffList = kOffMap + BM * kMapPitch;
    static constexpr int kSmem = kOffList + (kObs + K) * 2;
    static_assert(XS % 4 == 0 && kOffList % 8 == 0, "alignment");
};
__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

template <int TM, int G, int WU, int UL>
__global__ void __launch_bounds__(32 * kEncWarps, 2)
k_encoder_fp32(const uint8_t* rec, const float* __restrict__ W_enc, const float* __restrict__ b_enc, const uint32_t* odd_weights,
               float* __restrict__ h_out, int n, int H, int w_aligned, int early) {
    using E = Enc<TM, G, WU, UL>;
    static_assert(UL == 4 || (UL == 1 && TM == 1 && G == 1), "tiles");
    constexpr int BM = E::BM, BU = E::BU, XS = E::XS, K = E::K, S = E::S, R = E::R, D = G == 1 ? 2 : S == 3 ? 1 : 0;   // D: stages filled behind one before it is handed over
    constexpr int FULL = 1, EMPTY = FULL + S;   // barrier ids
    static_assert(EMPTY + S <= 16, "barriers");
    extern __shared__ __align__(16) float sm[];   // x [R][XS], w [R][BU], the records' map bytes [BM][kMapPitch], the list of features
    __shared__ uint32_t part[kEncWarps][4 * kMapRounds];
    float* const xring = sm;
    float* const wring = sm + R * XS;
    uint8_t* const map = reinterpret_cast<uint8_t*>(sm) + E::kOffMap;
    uint16_t* const list = reinterpret_cast<uint16_t*>(reinterpret_cast<uint8_t*>(sm) + E::kOffList);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int e0 = blockIdx.x * BM, u0 = blockIdx.y * BU;
    if (early & kLaunchNext) launch_next_kernel();
    wait_for_previous_kernel();
    // The map bytes of the block's envs (where there are none, the last one's again, which changes nothing), and which of them are not
    // zero in all envs: a bit a feature, 32 to a group
    {
        constexpr int ROWS = (BM + kEncWarps - 1) / kEncWarps, AT_ONCE = ROWS <= 9 ? ROWS : (ROWS + 1) / 2;   // a warp's envs; of them loaded before the first is stored
        uint32_t any[kMapRounds] = {};
#pragma unroll 1
        for (int i0 = warp; i0 < BM; i0 += AT_ONCE * kEncWarps) {
            uint32_t v[AT_ONCE][kMapRounds];
#pragma unroll
            for (int i = 0; i < AT_ONCE; i++) {
                const uint32_t* r = reinterpret_cast<const uint32_t*>(rec + (size_t)min(e0 + i0 + i * kEncWarps, n - 1) * kRec) + lane;
#pragma unroll
                for (int j = 0; j < kMapRounds; j++) v[i][j] = 32 * j + lane < kMap / 4 ? ld_now(r + 32 * j) : 0u;
            }
#pragma unroll
            for (int i = 0; i < AT_ONCE; i++) {
                if (i0 + i * kEncWarps >= BM) break;
                uint32_t* m = reinterpret_cast<uint32_t*>(map + (i0 + i * kEncWarps) * kMapPitch) + lane;
#pragma unroll
                for (int j = 0; j < kMapRounds; j++) {
                    any[j] |= v[i][j];
                    if (32 * j + lane < kMap / 4) m[32 * j] = v[i][j];
                }
            }
        }
        const bool all = __any_sync(0xffffffffu, (ld_now(odd_weights + lane) | ld_now(odd_weights + lane + 32)) != 0);
#pragma unroll
        for (int j = 0; j < kMapRounds; j++) {
            // a byte's bit 0 to bit 28 + its number, then to its place in the group
            uint32_t b = (((__vcmpne4(any[j], 0u) & 0x01010101u) * 0x10204080u) >> 28) << (4 * (lane & 7));
            if (all) b = 0xFu << (4 * (lane & 7));
#pragma unroll
            for (int d = 1; d < 8; d *= 2) b |= __shfl_xor_sync(0xffffffffu, b, d);
            if ((lane & 7) == 0) part[warp][4 * j + (lane >> 3)] = b;
        }
    }
    __syncthreads();
    // the list: lane c counts group c, then every warp writes some groups
    int total;
    {
        uint32_t rows = 0u;
        if (lane < kMapGroups) {
#pragma unroll
            for (int w = 0; w < kEncWarps; w++) rows |= part[w][lane];
            if (lane == kMapGroups - 1) rows &= ~0u >> (kMapGroups * 32 - kMap);
        } else if (lane < kGroups) {
            rows = ~0u >> (lane == kGroups - 1 ? (kGroups - kMapGroups) * 32 - kTail : 0);
        }
        int pos = __popc(rows);
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const int before = __shfl_up_sync(0xffffffffu, pos, d);
            if (lane >= d) pos += before;
        }
        total = __shfl_sync(0xffffffffu, pos, 31);
        pos -= __popc(rows);
#pragma unroll
        for (int i = 0; i < (kGroups + kEncWarps - 1) / kEncWarps; i++) {   // (groups from kGroups on have no bits)
            const int c = warp + i * kEncWarps;
            const uint32_t r = __shfl_sync(0xffffffffu, rows, c);
            const int p = __shfl_sync(0xffffffffu, pos, c);
            if (r >> lane & 1u) list[p + __popc(r & ((1u << lane) - 1u))] = (uint16_t)(c < kMapGroups ? 32 * c + lane : kMap + 32 * (c - kMapGroups) + lane);
        }
        if (warp == 0 && lane < K) list[total + lane] = 0;   // (a stage's end: copied, and not multiplied)
    }
    __syncthreads();
    const int stages = (total + K - 1) / K;
    if (warp >= kEncWarps - kEncFill) {
        // a warp has KW rows of every stage: their weights WR rows an instruction, a lane 16 bytes, their features XR rows an instruction, a lane an env
        constexpr int KW = K / kEncFill, WL = BU / 4, WR = 32 / WL, XL = BM < 32 ? BM : 32, XR = 32 / XL, ENVS = (BM + 31) / 32;
        static_assert(KW % 4 == 0 && BU <= 128 && 32 % WL == 0 && 32 % XL == 0 && KW % WR == 0 && KW % XR == 0, "whole rows");
        const int k0 = (warp - (kEncWarps - kEncFill)) * KW, xl = lane % XL;
        const bool whole = total == kObs;   // the list is all features
        const float* const wsrc = W_enc + u0 + 4 * (lane % WL);
        for (int i = 0; i < stages + D; i++) {
            if (i < stages) {
                const int s = i % S;
                if (i >= S) bar_sync(EMPTY + s, 32 * kEncWarps);
                const uint16_t* const rows = list + i * K + k0;
                float* const x = xring + (s * K + k0 + lane / XL) * XS + xl;
                float* const w = wring + (s * K + k0) * BU + 4 * lane;
                int f[KW / WR], g[KW / XR];   // the features whose weights and whose values this lane brings
                if constexpr (XR == 1) {
#pragma unroll
                    for (int k = 0; k < KW; k += 4) {
                        const uint2 v = *reinterpret_cast<const uint2*>(rows + k);
                        g[k] = v.x & 0xFFFFu; g[k + 1] = v.x >> 16; g[k + 2] = v.y & 0xFFFFu; g[k + 3] = v.y >> 16;
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < KW / XR; k++) g[k] = rows[k * XR + lane / XL];
                }
#pragma unroll
                for (int k = 0; k < KW / WR; k++) f[k] = WR == XR ? g[k] : rows[k * WR + lane / WL];
                if (w_aligned)
#pragma unroll
                    for (int k = 0; k < KW / WR; k++) copy16(w + k * WR * BU, wsrc + (size_t)f[k] * H, true, true);
                else
#pragma unroll
                    for (int k = 0; k < KW / WR; k++) copy16(w + k * WR * BU, wsrc + (size_t)f[k] * H, true, false);
                const bool maps = (i + 1) * K <= total - kTail;
                if (XR == 1 && whole && maps) {   // four features a word
                    uint32_t v[KW / 4][ENVS];
#pragma unroll
                    for (int q = 0; q < ENVS; q++) {
                        const uint8_t* m = map + (BM % 32 != 0 ? min(32 * q + lane, BM - 1) : 32 * q + lane) * kMapPitch + i * K + k0;
#pragma unroll
                        for (int k = 0; k < KW / 4; k++) v[k][q] = *reinterpret_cast<const uint32_t*>(m + 4 * k);
                    }
#pragma unroll
                    for (int q = 0; q < ENVS; q++)
                        if (BM % 32 == 0 || 32 * q + lane < BM)
#pragma unroll
                            for (int k = 0; k < KW; k++) x[k * XS + 32 * q] = (float)(v[k / 4][q] >> (8 * (k % 4)) & 0xFFu);
                } else if (maps) {
                    uint32_t v[KW / XR][ENVS];
#pragma unroll
                    for (int q = 0; q < ENVS; q++) {
                        const uint8_t* m = map + (BM > 32 && BM % 32 != 0 ? min(32 * q + lane, BM - 1) : 32 * q + xl) * kMapPitch;
#pragma unroll
                        for (int k = 0; k < KW / XR; k++) v[k][q] = m[g[k]];
                    }
#pragma unroll
                    for (int q = 0; q < ENVS; q++)
                        if (BM <= 32 || BM % 32 == 0 || 32 * q + lane < BM)
#pragma unroll
                            for (int k = 0; k < KW / XR; k++) x[k * XR * XS + 32 * q] = (float)v[k][q];
                } else {
#pragma unroll
                    for (int q = 0; q < ENVS; q++) {
                        const int e = 32 * q + xl;
                        if (BM > 32 && BM % 32 != 0 && e >= BM) break;
                        const uint8_t* const r = rec + (size_t)min(e0 + e, n - 1) * kRec + kMap;
#pragma unroll
                        for (int k = 0; k < KW / XR; k++) {
                            float* const to = x + k * XR * XS + 32 * q;
                            if (g[k] < kMap) *to = (float)map[e * kMapPitch + g[k]];
                            else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(r + 4 * (g[k] - kMap)) : "memory");
                        }
                    }
                }
            }
            copy_commit();
            copy_wait<D>();   // stage i - D is complete
            if (i >= D) bar_arrive(FULL + (i - D) % S, 32 * kEncWarps);
        }
        return;
    }
    const int el = warp % E::WM * UL * TM, ul = warp / E::WM * 32 * G + lane % (32 / UL) * UL, lg = lane / (32 / UL);   // the warp's first env
    float z1 = UL == 1 ? b_enc[u0 + ul] : 0.0f;   // the sum of a lane with one
    uint64_t z[G][TM][2];
#pragma unroll
    for (int g = 0; g < G; g++) {
        if (UL == 1) break;
        const float* b = b_enc + u0 + ul + 32 * g;
#pragma unroll
        for (int e = 0; e < TM; e++) { z[g][e][0] = f2pack(b[0], b[1]); z[g][e][1] = f2pack(b[2], b[3]); }
    }
    auto step = [&](const float* xp, const float* wp) {
        if constexpr (UL == 1) {
            z1 = fmaf(*xp, *wp, z1);
            return;
        }
        Frag<TM> x;
        x.load(xp, lg);
#pragma unroll
        for (int g = 0; g < G; g++) {
            const float4 w = *reinterpret_cast<const float4*>(wp + 32 * g);
            const uint64_t w01 = f2pack(w.x, w.y), w23 = f2pack(w.z, w.w);
#pragma unroll
            for (int e = 0; e < TM; e++) {
                z[g][e][0] = f2fma(x.v[e], w01, z[g][e][0]);
                z[g][e][1] = f2fma(x.v[e], w23, z[g][e][1]);
            }
        }
    };
    for (int i = 0; i < stages; i++) {
        const int s = i % S, left = total - i * K;
        const float* xp = xring + s * K * XS + el;
        const float* wp = wring + s * K * BU + ul;
        bar_sync(FULL + s, 32 * kEncWarps);
        if (left >= K) {
#pragma unroll
            for (int k = 0; k < K; k++) step(xp + k * XS, wp + k * BU);
        } else {
            for (int k = 0; k < left; k++) step(xp + k * XS, wp + k * BU);
        }
        if (i + S < stages) bar_arrive(EMPTY + s, 32 * kEncWarps);
    }
    if constexpr (UL == 1) {
        if (e0 + el < n) h_out[act_at(e0 + el, u0 + ul, H)] = z1;
        return;
    }
#pragma unroll
    for (int p = 0; p < Envs<TM>::kParts; p++) {
        const int env = e0 + el + Envs<TM>::at(p, lg);
        if (env >= n) continue;
#pragma unroll
        for (int i = 0; i < 4 * G; i++) {
            const int g = i >> 2, u = i & 3;
            float h[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                if (e >= Envs<TM>::count(p)) break;
                float lo, hi;
                f2unpack(z[g][Envs<TM>::first(p) + e][u >> 1], lo, hi);
                h[e] = (u & 1) ? hi : lo;
            }
            store_envs(h_out + act_at(env, u0 + ul + 32 * g + u, H), h, Envs<TM>::count(p));
        }
    }
}

// ---------------------------------------------------------------- classic game
// Record -> 1345 features, reference expand_obs_kernel (craftax_classic.cu:1265-1301).
__global__ void k_classic_expand(const uint8_t* __restrict__ rec, float* __restrict__ out, int n) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    const uint8_t* c = rec + (size_t)e * kClassicRec;
    float* o = out + (size_t)e * kClassicObs;
    int k = 0;
    for (int cell = 0; cell < kClassicCells; cell++) {
        const int8_t blk = (int8_t)c[cell];
        for (int b = 0; b < kClassicBlocks; b++) o[k++] = (blk == b) ? 1.0f : 0.0f;
        const uint8_t m = c[kClassicCells + cell];
        for (int j = 0; j < 4; j++) o[k++] = (m & (1 << j)) ? 1.0f : 0.0f;
    }
    int i2 = 2 * kClassicCells;
    for (int j = 0; j < kClassicInv + 4; j++) o[k++] = (float)(int8_t)c[i2++] / 10.0f;
    const int8_t dir = (int8_t)c[i2++];
    for (int d = 1; d <= 4; d++) o[k++] = (dir == d) ? 1.0f : 0.0f;
    const uint8_t sleeping = c[i2++];
    float light;
    memcpy(&light, c + i2, 4);
    o[k++] = light;
    o[k++] = sleeping ? 1.0f : 0.0f;
}

// Gather encoder in the order of the reference's encode_obs_kernel (craftax_classic.cu:1714-1751):
// bias, then per cell the block column and the set mob bits, then the 22 scalar features, every
// term as fmaf(x, W, acc).  One thread per (env, unit); the block's threads read a W_enc row
// coalesced.  Block ids outside [0,16] (never written by the game) are skipped.
__global__ void k_classic_encoder_fp32(const uint8_t* rec, const float* __restrict__ W_enc,
                                       const float* __restrict__ b_enc, float* __restrict__ h_out,
                                       int n, int H) {
    __shared__ uint8_t rs[kClassicRec];
    const int e = blockIdx.x;
    const int k = threadIdx.x;
    wait_for_previous_kernel();
    for (int i = threadIdx.x; i < kClassicRec; i += blockDim.x) rs[i] = rec[(size_t)e * kClassicRec + i];
    __syncthreads();
    const float* Wk = W_enc + k;
    float hv = b_enc[k];
    for (int cell = 0; cell < kClassicCells; cell++) {
        const int blk = (int8_t)rs[cell];
        if (blk >= 0 && blk < kClassicBlocks)
            hv = fmaf(1.0f, Wk[(size_t)(cell * (kClassicBlocks + 4) + blk) * H], hv);
        const uint8_t m = rs[kClassicCells + cell];
        const int fm = cell * (kClassicBlocks + 4) + kClassicBlocks;
        for (int j = 0; j < 4; j++)
            if (m & (1 << j)) hv = fmaf(1.0f, Wk[(size_t)(fm + j) * H], hv);
    }
    int oi = 2 * kClassicCells;
    int f = kClassicCells * (kClassicBlocks + 4);
    for (int j = 0; j < kClassicInv + 4; j++, f++)
        hv = fmaf((float)(int8_t)rs[oi++] / 10.0f, Wk[(size_t)f * H], hv);
    const int8_t dir = (int8_t)rs[oi++];
    for (int d = 1; d <= 4; d++, f++) hv = fmaf((dir == d) ? 1.0f : 0.0f, Wk[(size_t)f * H], hv);
    const uint8_t sleeping = rs[oi++];
    float light;
    memcpy(&light, rs + oi, 4);
    hv = fmaf(light, Wk[(size_t)f * H], hv);
    f++;
    hv = fmaf(sleeping ? 1.0f : 0.0f, Wk[(size_t)f * H], hv);
    h_out[act_at(e, k, H)] = hv;   // the scattered words meet in L2 (a record gathers 100 rows of W_enc)
}

// r_done int8 flags of the classic rollout (main_classic.cu:436-443) -> the float flags the
// MinGRU kernel takes
__global__ void k_done_to_terminals(const int8_t* __restrict__ done, float* __restrict__ out, int n) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < n) out[e] = done[e] != 0 ? 1.0f : 0.0f;
}

// ---------------------------------------------------------------- MinGRU layer
// d[i] = 1.0f / d[i] for d >= 1, n values at once (n is a constant once unrolled).  The compiler's correctly rounded division has a branch, so
// sigmoids written one by one run one after the other, about 150 cycles each: the 96 of a lane took half as long as a lone block's sums
// at hidden 256.  Here the reciprocals are refined without a branch, by a Newton step with the remainder in one FMA (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", 1990).  That this rounds correctly depends on the
// approximation that it starts from: k_selftest_reciprocals compares all values up to 2^126 with the division.  Beyond, and for infinity, where
// the reciprocal is subnormal or zero, the batch is divided.
constexpr int kReciprocals = 12;   // of a batch in the wide layers: three gates of four envs
template <int N> __device__ __forceinline__ void reciprocals(float (&d)[N], int n) {
    float r[N], most = 1.0f;
#pragma unroll
    for (int i = 0; i < N; i++) {
        if (i >= n) break;
        float a;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(d[i]));
        r[i] = fmaf(a, fmaf(-d[i], a, 1.0f), a);
        most = fmaxf(most, d[i]);
    }
    if (most > 0x1p126f)
#pragma unroll
        for (int i = 0; i < N; i++)
            if (i < n) r[i] = 1.0f / d[i];
#pragma unroll
    for (int i = 0; i < N; i++)
        if (i < n) d[i] = r[i];
}
// Denominators with the bits first .. last, in batches as the layers have them; where `far` is not zero it is the last of every batch.  Counts
// those whose reciprocal is not 1.0f / d.
__global__ void k_selftest_reciprocals(uint32_t first, uint32_t last, uint32_t far, unsigned long long* differing) {
    const uint32_t own = far != 0u ? kReciprocals - 1 : kReciprocals, stride = gridDim.x * blockDim.x;
    const uint32_t batches = (last - first) / own + 1;
    unsigned long long bad = 0;
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < batches; b += stride) {
        float d[kReciprocals], r[kReciprocals];
#pragma unroll
        for (uint32_t i = 0; i < kReciprocals; i++)
            r[i] = d[i] = __uint_as_float(i < own ? min(first + b * own + i, last) : far);
        reciprocals(r, kReciprocals);
#pragma unroll
        for (int i = 0; i < kReciprocals; i++) {
            const float want = 1.0f / d[i];
            if (__float_as_uint(r[i]) != __float_as_uint(want) && !(r[i] != r[i] && want != want)) bad++;
        }
    }
    if (bad != 0) atomicAdd(differing, bad);
}
// N values 1 / (1 + exp(-z)) at once
template <int N> __device__ __forceinline__ void sigmoids_ref(float (&z)[N], int n) {
#pragma unroll
    for (int i = 0; i < N; i++)
        if (i < n) z[i] = 1.0f + expf(-z[i]);
    reciprocals(z, n);
}
// The cell of an env and unit (k_mingru_epi_fwd, craftax_full.cu:9350-9395): zh is the first gate's sum, s[0 .. 2] the sigmoids of all three, x the layer's
// input, state is replaced; returns the layer's output.  One place for all layer kernels, whose batches must give the same bits.
__device__ __forceinline__ float cell(float zh, const float* s, float x, float& state) {
    const float gh = zh >= 0.0f ? zh + 0.5f : s[0];
    state = state + s[1] * (gh - state);
    return s[2] * state + (1.0f - s[2]) * x;
}

// One layer: gate dots (ascending j, fmaf) + cell.
// Wt is the layer's gate matrix as k_transpose_gates lays it out, x_in and h_out activations.  K chunks of 32; ST buffers:
// two where several blocks share an SM, more for small batches, which wait for the loads (chunks of 16 with three: 155 against
// 152 us a forward at 4,096 envs, 970 against 944 us at 8,192 envs with hidden 512, depth 3); the k loop has to be unrolled
// well (by 4: 170 us), but not whole (8,192 envs, hidden 512: 2 % slower).  Bound by the FMA pipe.  Two blocks an SM, so that blocks of five envs
// a lane and more keep everything in registers (three: 160 bytes of spills, 142 against 136 us at 4,096 envs).  us a forward, before the cell's loads and
// divisions were taken out of their chains and the heights followed the number of blocks, and now: 4,096 envs, hidden 256, depth 2 146.9 and 123.7;
// 5,120 222.1 and 153.9; 1,024 66.1 and 58.8; 8,192 envs, hidden 512, depth 3 887 and 827.
constexpr int kGruK = 32;
template <int TM, int WM, int WU> constexpr int gru_stage_floats() { return kGruK * (4 * TM * WM + 3 * 32 * WU); }

template <int TM, int WM, int WU, int ST>
__global__ void __launch_bounds__(32 * WM * WU, TM > 4 ? 2 : 3)
k_mingru_fp32(const float* x_in, const float* __restrict__ Wt, float* __restrict__ state,
              const float* prev_terminals, float* __restrict__ h_out, float* __restrict__ r_state,
              int r_bf16, int n, int H, int s_aligned, int early) {
    constexpr int T = 32 * WM * WU, BM = 4 * TM * WM, BU = 32 * WU, kStage = gru_stage_floats<TM, WM, WU>();
    using E = Envs<TM>;
    extern __shared__ __align__(16) float sm[];   // per stage: x [kGruK][BM], w [kGruK][3][BU]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int e0 = blockIdx.x * BM, u0 = blockIdx.y * BU;
    const int el = (warp % WM) * 4 * TM, ul = (warp / WM) * 32 + (lane & 7) * 4, lg = lane >> 3;   // the warp's first env
    const float* wsrc = Wt + (size_t)u0 * 3 * H;
    // the copies of a chunk, in pieces of 16 bytes a thread
    constexpr int NW = kGruK * 3 * BU / (4 * T), NX = (kGruK * (BM / 4) + T - 1) / T;
    static_assert(NW * 4 * T == kGruK * 3 * BU, "whole pieces");
    auto copy_w = [&](int c, int i) {
        const int at = 4 * (i * T + tid);
        copy16(sm + (c % ST) * kStage + kGruK * BM + at, wsrc + (size_t)c * kGruK * 3 * BU + at, true, true);
    };
    auto copy_x = [&](int c, int i) {
        const int at = i * T + tid;
        if (NX * T != kGruK * (BM / 4) && at >= kGruK * (BM / 4)) return;
        const int k = at / (BM / 4), env = e0 + 4 * (at % (BM / 4));
        const bool on = env < n;   // (n is a multiple of 32)
        copy16(sm + (c % ST) * kStage + 4 * at, x_in + act_at(on ? env : e0, c * kGruK + k, H), on, true);
    };
    if (early & kLaunchNext) launch_next_kernel();
    const int chunks = H / kGruK;
    if (!(early & kWeightsReady)) wait_for_previous_kernel();
#pragma unroll
    for (int c = 0; c < ST - 1; c++)
        if (c < chunks)
#pragma unroll
            for (int i = 0; i < NW; i++) copy_w(c, i);
    wait_for_previous_kernel();
#pragma unroll
    for (int c = 0; c < ST - 1; c++) {
        if (c < chunks)
#pragma unroll
            for (int i = 0; i < NX; i++) copy_x(c, i);
        copy_commit();
    }
#pragma unroll
    for (int p = 0; p < E::kParts; p++) {   // this lane's states, on their way to L2 while the sums run
        const int env = e0 + el + E::at(p, lg);
        if (env < n)
#pragma unroll
            for (int e = 0; e < E::count(p); e++)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(state + (size_t)(env + e) * H + u0 + ul));
    }
    uint64_t z[3][TM][2];
#pragma unroll
    for (int g = 0; g < 3; g++)
#pragma unroll
        for (int e = 0; e < TM; e++) z[g][e][0] = z[g][e][1] = 0ull;
    for (int c = 0; c < chunks; c++) {
        copy_wait<ST - 2>();
        __syncthreads();   // chunk c is complete, and everybody is done with chunk c - 1
        if (c + ST - 1 < chunks) {
#pragma unroll
            for (int i = 0; i < NW; i++) copy_w(c + ST - 1, i);
#pragma unroll
            for (int i = 0; i < NX; i++) copy_x(c + ST - 1, i);
        }
        copy_commit();
        const float* x = sm + (c % ST) * kStage + el;
        const float* w = sm + (c % ST) * kStage + kGruK * BM + ul;
#pragma unroll 16
        for (int k = 0; k < kGruK; k++) {
            Frag<TM> xv;
            xv.load(x + k * BM, lg);
#pragma unroll
            for (int g = 0; g < 3; g++) {
                const float4 wv = *reinterpret_cast<const float4*>(w + (k * 3 + g) * BU);
                const uint64_t w01 = f2pack(wv.x, wv.y), w23 = f2pack(wv.z, wv.w);
#pragma unroll
                for (int e = 0; e < TM; e++) {
                    z[g][e][0] = f2fma(w01, xv.v[e], z[g][e][0]);
                    z[g][e][1] = f2fma(w23, xv.v[e], z[g][e][1]);
                }
            }
        }
    }
    // The cell, a part of the lane's envs at a time: their states, flags and the inputs of the lane's units are loaded before anything is
    // done with them, those of the next part when half of the accumulators of this one are used up.
    float st[2][4][4], x[2][4][4], ended[2][4];
    auto fetch = [&](int p) {
        const int b = p & 1, env = e0 + el + E::at(p, lg);
        if (env >= n) return;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            if (e >= E::count(p)) break;
            const float* src = state + (size_t)(env + e) * H + u0 + ul;
            if (s_aligned) ld_now4(src, st[b][e]);
            else
#pragma unroll
                for (int u = 0; u < 4; u++) st[b][e][u] = src[u];
            ended[b][e] = prev_terminals != nullptr ? prev_terminals[env + e] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const float* src = x_in + act_at(env, u0 + ul + u, H);
            if (E::count(p) == 4) ld_now4(src, x[b][u]);
            else
#pragma unroll
                for (int e = 0; e < E::count(p); e++) x[b][u][e] = src[e];
        }
    };
    fetch(0);
#pragma unroll
    for (int p = 0; p < E::kParts; p++) {
        const int b = p & 1, env = e0 + el + E::at(p, lg), count = E::count(p);
        if (env >= n) {
            if (p + 1 < E::kParts) fetch(p + 1);
            continue;
        }
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (e < count && ended[b][e] != 0.0f) st[b][e][0] = st[b][e][1] = st[b][e][2] = st[b][e][3] = 0.0f;
        if (r_state != nullptr) {   // the post-zero state inputs
#pragma unroll
            for (int e = 0; e < 4; e++) {
                if (e >= count) break;
                const size_t o = (size_t)(env + e) * H + u0 + ul;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    if (r_bf16) reinterpret_cast<__nv_bfloat16*>(r_state)[o + u] = __float2bfloat16(st[b][e][u]);
                    else r_state[o + u] = st[b][e][u];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (u == 2 && p + 1 < E::kParts) fetch(p + 1);
            float h[4], zh[4], s[12];   // s: sigmoids of zh, zg, zp
#pragma unroll
            for (int e = 0; e < 4; e++)
#pragma unroll
                for (int g = 0; g < 3; g++) {
                    if (e >= count) break;
                    float lo, hi;
                    f2unpack(z[g][E::first(p) + e][u >> 1], lo, hi);
                    s[3 * e + g] = (u & 1) ? hi : lo;
                    if (g == 0) zh[e] = s[3 * e];
                }
            sigmoids_ref(s, 3 * count);
#pragma unroll
            for (int e = 0; e < 4; e++) {
                if (e >= count) break;
                h[e] = cell(zh[e], s + 3 * e, x[b][u][e], st[b][e][u]);
            }
            store_envs(h_out + act_at(env, u0 + ul + u, H), h, count);
        }
#pragma unroll
        for (int e = 0; e < 4; e++) {
            if (e >= count) break;
            float* dst = state + (size_t)(env + e) * H + u0 + ul;
            if (s_aligned) *reinterpret_cast<float4*>(dst) = make_float4(st[b][e][0], st[b][e][1], st[b][e][2], st[b][e][3]);
            else
#pragma unroll
                for (int u = 0; u < 4; u++) dst[u] = st[b][e][u];
        }
    }
}

// Small batches: N envs x N units a lane, N 1 or 2.  With 1 env x 4 units a lane the reads of shared memory (13 a k
// step and warp) are what a lone block waits for, 63 cycles a k step; here they are 4, or 8 for as many sums as those 13.  The sums are the same ones
// in the same order.  A block takes 2 N^2 envs x 64 units.
constexpr int kSmallUnits = 64, kSmallStages = 4, kSmallThreads = 128;
template <int N> struct Small {
    static constexpr int kEnvs = 2 * N * N, kStage = kGruK * (kEnvs + 3 * kSmallUnits);   // floats: x [kGruK][kEnvs], w [kGruK][3][64]
};
template <int N>
__global__ void __launch_bounds__(kSmallThreads)
k_mingru_small(const float* x_in, const float* __restrict__ Wt, float* __restrict__ state, const float* prev_terminals,
               float* __restrict__ h_out, float* __restrict__ r_state, int r_bf16, int H, int early) {
    constexpr int kEnvs = Small<N>::kEnvs, kStage = Small<N>::kStage;
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x, el = tid / (kSmallUnits / N) * N, u = tid % (kSmallUnits / N) * N;   // this lane's first env and unit
    const int e0 = blockIdx.x * kEnvs, u0 = blockIdx.y * kSmallUnits;   // (n is a multiple of 32)
    const float* wsrc = Wt + (size_t)u0 * 3 * H;
    constexpr int NW = kGruK * 3 * kSmallUnits / (4 * kSmallThreads), NX = kGruK * kEnvs / 2;   // pieces of 16 and of 8 bytes
    static_assert(NX <= kSmallThreads && kEnvs <= 32, "a thread a piece");
    auto copy_w = [&](int c) {
        float* w = sm + (c % kSmallStages) * kStage + kGruK * kEnvs;
#pragma unroll
        for (int i = 0; i < NW; i++) {
            const int at = 4 * (i * kSmallThreads + tid);
            copy16(w + at, wsrc + (size_t)c * kGruK * 3 * kSmallUnits + at, true, true);
        }
    };
    auto copy_x = [&](int c) {
        if (tid < NX)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(sm + (c % kSmallStages) * kStage + 2 * tid)),
                         "l"(x_in + act_at(e0 + 2 * tid % kEnvs, c * kGruK + 2 * tid / kEnvs, H)) : "memory");
    };
    if (early & kLaunchNext) launch_next_kernel();
    const int chunks = H / kGruK;
    if (!(early & kWeightsReady)) wait_for_previous_kernel();
#pragma unroll
    for (int c = 0; c < kSmallStages - 1; c++)
        if (c < chunks) copy_w(c);
    wait_for_previous_kernel();
#pragma unroll
    for (int c = 0; c < kSmallStages - 1; c++) {
        if (c < chunks) copy_x(c);
        copy_commit();
    }
    float st[N][N], ended[N], x_own[N][N], z[N][N][3] = {};
#pragma unroll
    for (int e = 0; e < N; e++) {
        ended[e] = prev_terminals != nullptr ? prev_terminals[e0 + el + e] : 0.0f;
#pragma unroll
        for (int i = 0; i < N; i++) {
            st[e][i] = state[(size_t)(e0 + el + e) * H + u0 + u + i];
            x_own[e][i] = x_in[act_at(e0 + el + e, u0 + u + i, H)];
        }
    }
    for (int c = 0; c < chunks; c++) {
        copy_wait<kSmallStages - 2>();
        __syncthreads();   // chunk c is complete, and everybody is done with chunk c - 1
        if (c + kSmallStages - 1 < chunks) {
            copy_w(c + kSmallStages - 1);
            copy_x(c + kSmallStages - 1);
        }
        copy_commit();
        const float* xs = sm + (c % kSmallStages) * kStage + el;
        const float* ws = sm + (c % kSmallStages) * kStage + kGruK * kEnvs + u;
        auto load = [](const float* p, float (&v)[N]) {
            if constexpr (N == 2) { const float2 f = *reinterpret_cast<const float2*>(p); v[0] = f.x; v[1] = f.y; }
            else v[0] = *p;
        };
#pragma unroll
        for (int k = 0; k < kGruK; k++) {
            float x[N], w[N];
            load(xs + k * kEnvs, x);
#pragma unroll
            for (int g = 0; g < 3; g++) {
                load(ws + (3 * k + g) * kSmallUnits, w);
#pragma unroll
                for (int e = 0; e < N; e++)
#pragma unroll
                    for (int i = 0; i < N; i++) z[e][i][g] = fmaf(w[i], x[e], z[e][i][g]);
            }
        }
    }
#pragma unroll
    for (int e = 0; e < N; e++)
#pragma unroll
        for (int i = 0; i < N; i++) {
            const size_t o = (size_t)(e0 + el + e) * H + u0 + u + i;
            float s = ended[e] != 0.0f ? 0.0f : st[e][i];
            const float zh = z[e][i][0];
            if (r_state != nullptr) {   // the post-zero state input
                if (r_bf16) reinterpret_cast<__nv_bfloat16*>(r_state)[o] = __float2bfloat16(s);
                else r_state[o] = s;
            }
            sigmoids_ref(z[e][i], 3);
            h_out[act_at(e0 + el + e, u0 + u + i, H)] = cell(zh, z[e][i], x_own[e][i], s);
            state[o] = s;
        }
}

// ---------------------------------------------------------------- heads
// logits_av[e][a] = bias[a] + sum_j W_av[a][j] * h[j][e] (ascending j); row A is the value head.
// Accumulator starts at the bias as in the scalar reference (craftax_full.cu:9838-9845).  A block
// takes 32 envs; a lane owns 2 envs x 3 rows, a warp 16 envs x 12 rows.  The 32 columns of h and the head
// matrix are staged in shared memory with every load in flight at once.
constexpr int kHeadEnvs = 32, kHeadRows = 12, kHeadLaneRows = 3;
constexpr int head_row_groups(int A) { return (A + 1 + kHeadRows - 1) / kHeadRows; }
constexpr int head_threads(int A) { return 64 * head_row_groups(A); }
constexpr size_t head_smem(int H, int A) {
    return ((size_t)kHeadEnvs * H + (size_t)head_row_groups(A) * kHeadRows * (H + 4)) * sizeof(float);
}

__global__ void __launch_bounds__(384) k_heads_fp32(const float* h, const float* __restrict__ W_a,
                                                    const float* __restrict__ b_a, const float* __restrict__ W_v,
                                                    const float* __restrict__ b_v, float* __restrict__ logits_av,
                                                    int n, int H, int A, int early) {
    extern __shared__ __align__(16) float hs[];   // h [H][32], then W [rows][H + 4]
    float* wsh = hs + kHeadEnvs * H;
    const int tid = threadIdx.x, T = blockDim.x, warp = tid >> 5, lane = tid & 31;
    const int e0 = blockIdx.x * kHeadEnvs, WS = H + 4;
    if (early & kLaunchNext) launch_next_kernel();
    if (!(early & kWeightsReady)) wait_for_previous_kernel();
    for (int a = warp; a < A + 1; a += T / 32) {
        const float* w = a < A ? W_a + (size_t)a * H : W_v;
        const bool al = (reinterpret_cast<uintptr_t>(w) & 15) == 0;
        for (int j = 4 * lane; j < H; j += 128) copy16(wsh + a * WS + j, w + j, true, al);
    }
    wait_for_previous_kernel();
    const float* hsrc = h + (size_t)e0 * H;   // 32 envs are one tile
    for (int i = 4 * tid; i < H * kHeadEnvs; i += 4 * T) copy16(hs + i, hsrc + i, true, true);
    copy_commit();
    const int a0 = (warp >> 1) * kHeadRows + (lane >> 3) * kHeadLaneRows, el = 16 * (warp & 1) + 2 * (lane & 7);
    float z[kHeadLaneRows][2];
#pragma unroll
    for (int r = 0; r < kHeadLaneRows; r++)
        z[r][0] = z[r][1] = a0 + r < A ? b_a[a0 + r] : b_v[0];
    copy_wait<0>();
    __syncthreads();
#pragma unroll 4
    for (int j = 0; j < H; j += 4) {
        float w[kHeadLaneRows][4];
#pragma unroll
        for (int r = 0; r < kHeadLaneRows; r++) {
            const float4 v = *reinterpret_cast<const float4*>(wsh + (a0 + r) * WS + j);
            w[r][0] = v.x; w[r][1] = v.y; w[r][2] = v.z; w[r][3] = v.w;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float2 x = *reinterpret_cast<const float2*>(hs + (j + q) * kHeadEnvs + el);
#pragma unroll
            for (int r = 0; r < kHeadLaneRows; r++) {
                z[r][0] = fmaf(w[r][q], x.x, z[r][0]);
                z[r][1] = fmaf(w[r][q], x.y, z[r][1]);
            }
        }
    }
    __syncthreads();   // the h columns are used up: the logits take their place
#pragma unroll
    for (int r = 0; r < kHeadLaneRows; r++)
#pragma unroll
        for (int e = 0; e < 2; e++)
            if (a0 + r < A + 1) hs[(el + e) * (A + 1) + a0 + r] = z[r][e];
    __syncthreads();
    for (int i = tid; i < kHeadEnvs * (A + 1); i += T) logits_av[(size_t)e0 * (A + 1) + i] = hs[i];
}

// ---------------------------------------------------------------- sampler
// k_value_sample (craftax_full.cu:9714-9741); logits already carry their biases.  A block of 128
// threads takes 32 envs: the rows come in coalesced, four threads of an env take its maximum and its
// exponentials (both independent of order), one thread adds them up in the reference's order.
// The running sums are kept, so that the search for the first one that reaches the target is parallel too.
// `ctr` (optional): device step counter {offset, blocks finished}; with `bump` the last block that has read it raises it.
constexpr int kSampleEnvs = 32, kSampleThreads = 128;

__global__ void __launch_bounds__(kSampleThreads)
k_sample(const float* logits, int ld, int A, const float* uniforms, uint64_t seed,
         uint64_t env_offset, unsigned long long* ctr, int bump, int n, float* __restrict__ env_actions,
         int32_t* __restrict__ actions, float* __restrict__ logprobs, float* __restrict__ values, int early) {
    __shared__ float l[kSampleEnvs][kMaxActions + 2], p[kSampleEnvs + 1][kMaxActions + 2];   // odd row length
    const int tid = threadIdx.x, e0 = blockIdx.x * kSampleEnvs;
    const int cols = values != nullptr ? A + 1 : A;
    if (early & kLaunchNext) launch_next_kernel();
    wait_for_previous_kernel();
    const int envs = min(kSampleEnvs, n - e0);
    for (int i = tid; i < envs * cols; i += kSampleThreads)
        l[i / cols][i % cols] = logits[(size_t)(e0 + i / cols) * ld + i % cols];
    const int e = tid >> 2, part = tid & 3;   // env and quarter of its actions
    const unsigned mates = 0xFu << (tid & 28);
    float u = 0.0f;
    if (part == 0 && e < envs)
        u = uniforms != nullptr ? uniforms[e0 + e]
                                : philox_uniform(seed, env_offset + (uint64_t)(e0 + e), ctr ? *ctr : 0ULL);
    __syncthreads();   // the rows are here, and this block has read the counter
    if (bump && tid == kSampleThreads - 1) {
        if (gridDim.x > 1) __threadfence();
        if (gridDim.x == 1 || atomicAdd(ctr + 1, 1ULL) == gridDim.x - 1) {
            ctr[0] += 1ULL;
            ctr[1] = 0ULL;
        }
    }
    if (e >= envs) return;   // (all four threads of an env)
    float m = -INFINITY;
#pragma unroll 4
    for (int a = part; a < A; a += 4) m = fmaxf(m, l[e][a]);
    m = fmaxf(m, __shfl_xor_sync(mates, m, 1));
    m = fmaxf(m, __shfl_xor_sync(mates, m, 2));
#pragma unroll 4
    for (int a = part; a < A; a += 4) p[e][a] = expf(l[e][a] - m);
    __syncwarp(mates);
    float total = 0.0f;
    if (part == 0) {
        for (int a = 0; a < A; a += 8) {   // (loads of a batch before its stores)
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = p[e][a + i];   // beyond A: room in the row's neighbours, not used
#pragma unroll
            for (int i = 0; i < 8; i++) {
                if (a + i >= A) break;
                total += v[i];
                p[e][a + i] = total;
            }
        }
    }
    __syncwarp(mates);
    total = __shfl_sync(mates, total, tid & 28);
    u = __shfl_sync(mates, u, tid & 28);
    const float target = u * total;
    int action = A - 1;
    for (int a = part; a < A; a += 4)
        if (target <= p[e][a]) { action = a; break; }
    action = min(action, __shfl_xor_sync(mates, action, 1));
    action = min(action, __shfl_xor_sync(mates, action, 2));
    if (part == 0) {
        const int env = e0 + e;
        if (env_actions) env_actions[env] = (float)action;
        if (actions) actions[env] = action;
        if (logprobs) logprobs[env] = l[e][action] - m - logf(total);
        if (values) values[env] = l[e][A];
    }
}

// The same for a large batch of logits by itself: a thread an env, 128 envs a block, whose rows come in coalesced.  Four
// threads an env fill the GPU with a quarter of the envs, and with few actions most of what they do is waiting.
// us with four threads / one: 262,144 envs 14.6 / 4.1 with 2 actions, 22.5 / 10.8 with 17, 42.8 / 30.8 with 43, 55.6 / 51.4 with
// 63; 65,536 envs 5.4 / 4.1, 8.0 / 6.8, 14.8 / 15.0, 18.6 / 20.4; 16,384 envs 3.4 / 4.1, 3.7 / 6.1, 6.1 / 13.6, 7.7 / 18.5.
constexpr int kSampleRows = 128;
__global__ void __launch_bounds__(kSampleRows)
k_sample_rows(const float* logits, int ld, int A, const float* uniforms, int n,
              int32_t* __restrict__ actions, float* __restrict__ logprobs) {
    extern __shared__ float rows[];   // [kSampleRows][A | 1]: logits, then the running sums of the exponentials
    const int tid = threadIdx.x, e0 = blockIdx.x * kSampleRows, pitch = A | 1;
    wait_for_previous_kernel();
    const int envs = min(kSampleRows, n - e0), step_e = kSampleRows / A, step_a = kSampleRows % A;
    for (int e = tid / A, a = tid % A; e < envs; e += step_e, a += step_a) {
        if (a >= A) {
            a -= A;
            if (++e >= envs) break;
        }
        rows[e * pitch + a] = logits[(size_t)(e0 + e) * ld + a];
    }
    __syncthreads();
    if (tid >= envs) return;
    float* p = rows + tid * pitch;
    const float u = uniforms[e0 + tid];
    float m = p[0], total = 0.0f;
    for (int a = 1; a < A; a++) m = fmaxf(m, p[a]);
    for (int a = 0; a < A; a++) {
        total += expf(p[a] - m);
        p[a] = total;
    }
    const float target = u * total;
    int action = 0;
    while (action < A - 1 && !(target <= p[action])) action++;
    actions[e0 + tid] = action;
    logprobs[e0 + tid] = logits[(size_t)(e0 + tid) * ld + action] - m - logf(total);
}

__global__ void k_uniforms(uint64_t seed, uint64_t env_offset, uint64_t step, int n, float* u) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < n) u[e] = philox_uniform(seed, env_offset + (uint64_t)e, step);
}

__global__ void k_fetch(const uint4* src, uint4* __restrict__ dst, size_t count) {
    wait_for_previous_kernel();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) dst[i] = src[i];
}

__global__ void k_bump(unsigned long long* ctr) { *ctr += 1ULL; }

// Gate matrices for the fp32 layer kernel: Wt[l][unit tile][j][gate][unit of the tile] = W[l][gate H + unit][j], tiles of 64
// units, or of 32 where the hidden size is an odd multiple of it.  The last kOddWords blocks look W_enc over, an equal share each,
// and leave behind the gate matrices whether anything in it is infinite or not a number (k_encoder_fp32).
__global__ void k_transpose_gates(const float* __restrict__ W, float* __restrict__ Wt, int H, int L, const float* __restrict__ W_enc, int enc) {
    const size_t per = (size_t)3 * H * H, idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int share = (int)blockIdx.x - (int)(gridDim.x - kOddWords);
    if (share >= 0) {
        bool odd = false;
        for (int i = share * (int)blockDim.x + threadIdx.x; i < enc; i += kOddWords * (int)blockDim.x) odd |= !(fabsf(W_enc[i]) < INFINITY);
        odd = __syncthreads_or(odd);
        if (threadIdx.x == 0) reinterpret_cast<uint32_t*>(Wt + per * L)[share] = odd ? 1u : 0u;
        return;
    }
    if (idx >= per * L) return;
    const size_t l = idx / per, r = (idx % per) / H, j = idx % H;
    const int U = H % 64 == 0 ? 64 : 32, g = (int)(r / H), u = (int)(r % H);
    Wt[l * per + (size_t)(u / U) * 3 * H * U + (j * 3 + g) * U + u % U] = W[idx];
}

// Reference initialiser: U(+-bound) from Philox(seed, subsequence, index)
// (k_nn_init_weights, craftax_full.cu:9123-9131).
__global__ void k_init_uniform(float* w, int count, float bound, uint64_t seed, int subseq) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    curandStatePhilox4_32_10_t st;
    curand_init(seed, (uint64_t)subseq, (uint64_t)i, &st);
    w[i] = (2.0f * curand_uniform(&st) - 1.0f) * bound;
}

// ---------------------------------------------------------------- launchers
int launch_expand(const uint8_t* rec, float* out, int n, cudaStream_t st) {
    size_t total = (size_t)n * kObs;
    k_expand<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(rec, out, n);
    CFX_CUDA(cudaGetLastError());
    return CFX_OK;
}

int launch_classic_expand(const uint8_t* rec, float* out, int n, cudaStream_t st) {
    k_classic_expand<<<(n + 127) / 128, 128, 0, st>>>(rec, out, n);
    CFX_CUDA(cudaGetLastError());
    return CFX_OK;
}

int launch_done_to_terminals(const int8_t* done, float* out, int n, cudaStream_t st) {
    k_done_to_terminals<<<(n + 255) / 256, 256, 0, st>>>(done, out, n);
    CFX_CUDA(cudaGetLastError());
    return CFX_OK;
}

int launch_sample(const float* logits, int ld, int A, const float* u, uint64_t seed,
                  uint64_t env_offset, unsigned long long* step_ctr, int bump, int n,
                  float* env_actions, int32_t* actions, float* logprobs, float* values,
                  cudaStream_t st, int early) {
    return launch_chained(k_sample, dim3((n + kSampleEnvs - 1) / kSampleEnvs), kSampleThreads, 0, st, logits, ld, A, u,
                          seed, env_offset, step_ctr, bump, n, env_actions, actions, logprobs, values, early);
}

int launch_sample_logits(const float* logits, int ld, int A, const float* u, int n, int32_t* actions, float* logprobs,
                         cudaStream_t st) {
    if (n < 65536 || (n < 131072 && A > 32))
        return launch_sample(logits, ld, A, u, 0, 0, nullptr, 0, n, nullptr, actions, logprobs, nullptr, st);
    return launch_chained(k_sample_rows, dim3((n + kSampleRows - 1) / kSampleRows), kSampleRows,
                          (size_t)kSampleRows * (A | 1) * sizeof(float), st, logits, ld, A, u, n, actions, logprobs);
}

int launch_uniforms(uint64_t seed, uint64_t env_offset, uint64_t step, int n, float* u, cudaStream_t st) {
    k_uniforms<<<(n + 255) / 256, 256, 0, st>>>(seed, env_offset, step, n, u);
    CFX_CUDA(cudaGetLastError());
    return CFX_OK;
}

int launch_fetch(const void* host, void* dst, size_t bytes, cudaStream_t st) {
    const size_t count = bytes / 16;
    return launch_chained(k_fetch, dim3((unsigned)((count + 127) / 128)), 128, 0, st, (const uint4*)host, (uint4*)dst, count);
}

int launch_bump(unsigned long long* ctr, cudaStream_t st) {
    k_bump<<<1, 1, 0, st>>>(ctr);
    CFX_CUDA(cudaGetLastError());
    return CFX_OK;
}

int launch_transpose_gates(const float* params, const ArenaLayout& o, float* Wt, int H, int L, cudaStream_t st) {
    size_t total = (size_t)L * 3 * H * H;
    k_transpose_gates<<<(unsigned)((total + 255) / 256) + kOddWords, 256, 0, st>>>(params + o.w_gru, Wt, H, L, params + o.w_enc, (int)(o.b_enc - o.w_enc));
    CFX_CUDA(cudaGetLastError());
    return CFX_OK;
}

int launch_init_uniform(float* w, int count, float bound, uint64_t seed, int subseq, cudaStream_t st) {
    k_init_uniform<<<(count + 255) / 256, 256, 0, st>>>(w, count, bound, seed, subseq);
    CFX_CUDA(cudaGetLastError());
    return CFX_OK;
}

int selftest_reciprocals(uint32_t first, uint32_t last, uint32_t far, uint64_t* differing) {
    unsigned long long* count = nullptr;
    CFX_CUDA(cudaMalloc((void**)&count, sizeof(*count)));
    cudaError_t e = cudaMemset(count, 0, sizeof(*count));
    if (e == cudaSuccess) {
        k_selftest_reciprocals<<<8 * kSMs, 256>>>(first, last, far, count);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(differing, count, sizeof(*count), cudaMemcpyDeviceToHost);
    cudaFree(count);
    CFX_CUDA(e);
    return CFX_OK;
}

// The tiles.  What a forward costs is the number of blocks that the fullest SM has one after the other, so the envs of a lane, TM, are
// those for which that number times the time of a block is the least; both are estimated from what blocks of each height take alone and two to an SM.
// What each height is for, us a forward with all of them and without it: layers, 5 (2,944 envs, hidden 256, depth 2) 98.7 and 103.9, 6 (1,760) 78.0 and 84.0,
// 7 (4,096) 123.6 and 128.1, 8 (8,192, hidden 512, depth 3) 827 and 864, 9 (2,656, hidden 512) 222 and 249.
static int sm_rounds(int n, int envs, int unit_tiles) { return ((n + envs - 1) / envs * unit_tiles + kSMs - 1) / kSMs; }
// Up to q = 32 a lane has one sum, or one of each gate (tile 0): us a forward of 32 envs, hidden 256, depth 2, with 4 units a lane in both kernels
// 46.2, in the encoder 38.7, in neither 32.0; 64 envs 47.6, 43.7 and 34.2; 128 envs 49.1 and 44.1; 192 envs 48.7 and 63; 32 envs, hidden 512 73 and 46;
// 256 envs, hidden 128 38.7 and 35.2; 512 envs, hidden 64 33.4 and 31.1.
constexpr int kSmallest = 32;
// A layer.  Tile 1 under q = 96, where even tiles of 4 envs leave schedulers without a warp: 2 envs x 2 units a lane (hidden sizes that are odd multiples
// of 32: 1 env x 4 units; us a forward, that and 2 x 2: 160 envs, hidden 256 48.2 and 44.5, 256 48.4 and 45.0, 320 71.4 and 62.2, 160 envs, hidden 512
// 106.3 and 86.7; from q = 96 to 592 2 x 2 and 4 x 4 take the same time).  Blocks of 4 envs a lane take the same time alone and beside each other, those
// of more envs a little less beside one.  Narrow layers have as much to do around the sums as in them, and stay with 4 longer (4,096 envs, hidden 128:
// 52.9 us, 54.3 with 7; 8,192 78.5 and 77.5).
static int strict_tile(int n, int H) {
    const long long q = (long long)n * H / 1024;
    if (q <= kSmallest && H % 64 == 0) return 0;
    if (q < 96) return 1;
    if (H % 64 != 0) return q >= 1024 ? 8 : 4;
    if (H < 256 && q < 1024) return 4;
    constexpr float kAlone[10] = {0, 0, 0, 0, 5.4f, 7.4f, 8.1f, 10.0f, 10.7f, 12.5f};
    int best = 0;
    float least = 0.0f;
    for (int tm = 4; tm <= 9; tm++) {
        const int b = sm_rounds(n, 8 * tm, H / 64);
        const float cost = kAlone[tm] * (tm == 4 ? (float)b : 1.83f * (b / 2) + b % 2);
        if (best == 0 || cost < least) { best = tm; least = cost; }
    }
    return best;
}
// The encoder: TM envs x 8 units a lane, where a block takes TM + 2 units of time, or, past the first round, TM + 4 where an SM holds one block at a time, whose
// first 3,000 cycles are then under no other's sums; 4 envs x 4 units as long as every block has an SM of its own (hidden 256, depth 1: 1,024 envs 42.9 us, 45.0
// with 8 units a lane; 1,536 56.3 and 48.9), 1 env x 4 units under q = 96.  Of the heights at 66 sizes, records of a game, this choice is the fastest or within 1.5 %
// of it, but for hidden 320 at 8,192 and 12,288 envs (2 and 4 %).  us with each of the heights 4 to 9, depth 1: 4,096 envs, hidden 256 78.0, 85.2, 91.3,
// 77.3, 81.0, 86.3; 6,144 112, 120, 110, 117, 124, 135; 65,536 936, 934, 931, 919, 911, 955; 10,656, hidden 128 86.8, 78.8, 85.0, 91.8, 96.6, 79.8;
// hidden 192, one round of blocks at 6,304 (9) 93.7, 91.5, 102.9, 113.7, 109.6, 92.1, several at 8,192 110, 121, 113, 124, 129, 141, 65,536 710, 704, 755, 761, 762, 782.
// With 9 a lane spills 12 or 32 bytes (128 registers, two blocks of 256 threads an SM).
struct EncoderTile { int tm, g; };
constexpr bool two_blocks(int tm, int wu) { return wu == 2 || tm <= 5; }   // (see strict_encoder)
static EncoderTile strict_encoder_tile(int n, int H) {
    const long long q = (long long)n * H / 1024;
    if (q <= kSmallest) return {0, 1};
    if (q < 96) return {1, 1};
    if (H % 64 != 0 || sm_rounds(n, 64, H / 32) == 1) return {4, 1};
    const int wu = H % 128 == 0 ? 2 : 1;
    int best = 4;
    auto cost = [&](int tm) {
        const int rounds = sm_rounds(n, 16 * tm / wu, H / (64 * wu));
        return rounds * (tm + (rounds > 1 && !two_blocks(tm, wu) ? 4 : 2));
    };
    for (int tm = 5; tm <= 9; tm++)
        if (cost(tm) < cost(best)) best = tm;
    return {best, 2};
}

// Layers with 4 envs a lane: three stages of weights where few blocks share an SM
static bool strict_deep(int n, int H) { return (long long)n * H / 1024 <= 592; }
void strict_tiles(int n, int H, int* layer, int* deep, int* encoder, int* groups) {
    const EncoderTile te = strict_encoder_tile(n, H);
    *layer = strict_tile(n, H);
    *deep = *layer == 4 && H % 64 == 0 && strict_deep(n, H);
    *encoder = te.tm;
    *groups = te.g;
}

template <int TM, int G, int WU, int UL = 4>
static int strict_encoder(const StrictArgs& a, const ArenaLayout& o, int early, cudaStream_t st) {
    using E = Enc<TM, G, WU, UL>;
    static_assert(two_blocks(TM, WU) == (2 * (E::kSmem + 2048) <= 228 * 1024), "what the rule for the tiles goes by");
    int rc = allow_smem<k_encoder_fp32<TM, G, WU, UL>, E::kSmem>();
    if (rc) return rc;
    return launch_chained(k_encoder_fp32<TM, G, WU, UL>, dim3((a.n + E::BM - 1) / E::BM, a.H / E::BU), 256, E::kSmem, st, a.records,
                          a.params + o.w_enc, a.params + o.b_enc, reinterpret_cast<const uint32_t*>(a.gates_t + strict_gate_floats(a.H, a.L) - kOddWords),
                          a.scratch_h[0], a.n, a.H, ((uintptr_t)(a.params + o.w_enc) & 15) == 0, early);
}

template <int TM, int WM, int WU, int ST>
static int strict_layers(const StrictArgs& a, int early, cudaStream_t st) {
    const int H = a.H, n = a.n;
    constexpr int BM = 4 * TM * WM, BU = 32 * WU, T = 32 * WM * WU;
    constexpr int smem = ST * gru_stage_floats<TM, WM, WU>() * (int)sizeof(float);
    int rc = allow_smem<k_mingru_fp32<TM, WM, WU, ST>, smem>();
    if (rc) return rc;
    const dim3 grid((n + BM - 1) / BM, H / BU);
    const int s_aligned = ((uintptr_t)a.state & 15) == 0;
    for (int l = 0; l < a.L; l++) {
        float* r = a.r_state ? reinterpret_cast<float*>(reinterpret_cast<char*>(a.r_state) +
                                                        (size_t)l * n * H * (a.r_state_bf16 ? 2 : 4))
                             : nullptr;
        rc = launch_chained(k_mingru_fp32<TM, WM, WU, ST>, grid, T, smem, st, a.scratch_h[l & 1],
                            a.gates_t + (size_t)l * 3 * H * H, a.state + (size_t)l * n * H, a.prev_terminals,
                            a.scratch_h[(l + 1) & 1], r, a.r_state_bf16, n, H, s_aligned, early);
        if (rc) return rc;
    }
    return CFX_OK;
}

// (H a multiple of 64)
template <int N>
static int strict_layers_small(const StrictArgs& a, int early, cudaStream_t st) {
    constexpr int smem = kSmallStages * Small<N>::kStage * (int)sizeof(float);
    int rc = allow_smem<k_mingru_small<N>, smem>();
    for (int l = 0; l < a.L && rc == CFX_OK; l++) {
        const size_t at = (size_t)l * a.n * a.H;
        float* r = a.r_state ? reinterpret_cast<float*>(reinterpret_cast<char*>(a.r_state) + at * (a.r_state_bf16 ? 2 : 4)) : nullptr;
        rc = launch_chained(k_mingru_small<N>, dim3(a.n / Small<N>::kEnvs, a.H / kSmallUnits), kSmallThreads, smem, st, a.scratch_h[l & 1],
                            a.gates_t + (size_t)l * 3 * a.H * a.H, a.state + at, a.prev_terminals, a.scratch_h[(l + 1) & 1], r, a.r_state_bf16,
                            a.H, early);
    }
    return rc;
}

template <int N> using Int = std::integral_constant<int, N>;
// Full strict forward.  scratch_h: two buffers of n H activations; logits_av [n][A+1].
int strict_forward(const StrictArgs& a, cudaStream_t st, int* launches) {
    const int H = a.H, L = a.L, A = a.A, n = a.n;
    const ArenaLayout o = ArenaLayout::make(H, L, A, a.game == CFX_GAME_CLASSIC ? kClassicObs : kObs);
    int rc;
    const long long q = (long long)n * H / 1024;
    const int tm = strict_tile(n, H);
    const EncoderTile te = strict_encoder_tile(n, H);
    // every kernel of a small forward lets the next one start at once, where all their blocks have SMs of their own (512 envs, 64 blocks a layer: 88 us
    // with it, 72 without; 32 envs, hidden 256, depth 2, 194 blocks: 34.4 and 31.6)
    auto count = [&](int tile) { return tile == 0 ? 8 * q : tile == 1 ? 2 * q : q / 2; };
    const long long blocks = count(te.tm) + L * count(tm) + n / 16;
    const int early = (a.game == CFX_GAME_FULL && te.tm <= 1 && blocks <= kSMs ? kLaunchNext : 0) | (a.weights_ready ? kWeightsReady : 0);
    if (a.game == CFX_GAME_CLASSIC) {
        rc = launch_chained(k_classic_encoder_fp32, dim3(n), H, 0, st, a.records, a.params + o.w_enc, a.params + o.b_enc,
                            a.scratch_h[0], n, H);
    } else {
        // (two warps side by side along the units, where there are 128: half of the conversions are other warps' too)
        auto encode = [&](auto tile) {
            constexpr int TM = decltype(tile)::value;
            return H % 128 == 0 ? strict_encoder<TM, 2, 2>(a, o, early, st) : strict_encoder<TM, 2, 1>(a, o, early, st);
        };
        if (te.tm == 0) rc = strict_encoder<1, 1, 1, 1>(a, o, early, st);
        else if (te.tm == 1) rc = strict_encoder<1, 1, 1>(a, o, early, st);
        else if (te.g == 1) rc = strict_encoder<4, 1, 1>(a, o, early, st);
        else rc = te.tm == 4 ? encode(Int<4>()) : te.tm == 5 ? encode(Int<5>()) : te.tm == 6 ? encode(Int<6>())
                  : te.tm == 7 ? encode(Int<7>()) : te.tm == 8 ? encode(Int<8>()) : encode(Int<9>());
    }
    if (rc) return rc;
    // a hidden size that is an odd multiple of 32 has the warps of a block side by side along the envs
    if (H % 64 != 0)
        rc = tm == 8 ? strict_layers<8, 4, 1, 2>(a, early, st) : tm == 4 ? strict_layers<4, 4, 1, 2>(a, early, st)
                                                                         : strict_layers<1, 4, 1, 4>(a, early, st);
    else if (tm == 0) rc = strict_layers_small<1>(a, early, st);
    else if (tm == 1) rc = strict_layers_small<2>(a, early, st);
    else if (tm == 4) rc = strict_deep(n, H) ? strict_layers<4, 2, 2, 3>(a, early, st) : strict_layers<4, 2, 2, 2>(a, early, st);
    else rc = tm == 5 ? strict_layers<5, 2, 2, 2>(a, early, st) : tm == 6 ? strict_layers<6, 2, 2, 2>(a, early, st)
              : tm == 7 ? strict_layers<7, 2, 2, 2>(a, early, st) : tm == 8 ? strict_layers<8, 2, 2, 2>(a, early, st)
                                                                         : strict_layers<9, 2, 2, 2>(a, early, st);
    if (rc) return rc;
    const size_t hsmem = head_smem(H, A);
    if ((rc = allow_smem<k_heads_fp32, (int)head_smem(kMaxHidden, kMaxActions)>())) return rc;
    rc = launch_chained(k_heads_fp32, dim3(n / kHeadEnvs), head_threads(A), hsmem, st, a.scratch_h[L & 1],
                        a.params + o.w_a, a.params + o.b_a, a.params + o.w_v, a.params + o.b_v, a.logits_av, n, H, A, early);
    if (rc) return rc;
    rc = launch_sample(a.logits_av, A + 1, A, a.uniforms, a.seed, a.env_offset, a.step_ctr, a.bump_step, n,
                       a.env_actions, a.actions, a.logprobs, a.values, st, early);
    if (rc) return rc;
    if (launches) *launches = 1 + L + 2;
    return CFX_OK;
}

}  // namespace cfx

// ---------------------------------------------------------------- allocation-free variant
// Strict fp32 forward whose scratch lives in a fixed device array instead of buffers from
// cudaMalloc.  Meant for hosts that must not allocate once they are running: a rollout
// worker embedded in another runtime that owns the whole device heap and hands out no
// memory, or a latency-bound loop where cudaMalloc's device-wide synchronisation (and its
// chance of failing on a fragmented heap hours into a run) is not acceptable.  Such a caller
// brings its own parameter arena, state, inputs and outputs; everything else is here.
//
// Limits: hidden = 256, layers <= 4, actions <= 63, num_envs <= 1024 (multiple of 32).
// The array (5.5 MB) is resident on every GPU that loads this library until the process
// exits.  All calls share it: two calls that overlap on the GPU (different streams, or
// different host threads) race on it; serialise them.  Nothing in it has to start at zero:
// the transposed gate matrices, both layer buffers and the logits are fully rewritten by
// each call before they are read, so stale contents of an earlier call are harmless.
namespace cfx {
constexpr int kStaticMaxEnvs = 1024, kStaticHidden = 256, kStaticMaxLayers = 4;
constexpr size_t kStaticGates = strict_gate_floats(kStaticHidden, kStaticMaxLayers);
constexpr size_t kStaticLayerBuf = (size_t)kStaticMaxEnvs * kStaticHidden;
constexpr size_t kStaticLogits = (size_t)kStaticMaxEnvs * (kMaxActions + 1);
constexpr size_t kStaticFloats = kStaticGates + 2 * kStaticLayerBuf + kStaticLogits;

static __device__ __align__(256) float g_static_scratch[kStaticFloats];

// Device address of the array per device ordinal; in host code the symbol's name is only a
// handle for cudaGetSymbolAddress, never a pointer a kernel could use.  The cache is filled
// once per device (atomic: two host threads may make their first calls together and resolve
// the same address).  It is not invalidated: after cudaDeviceReset the library must be
// reloaded before this entry point is used again.
constexpr int kStaticMaxDevices = 64;
static std::atomic<float*> g_static_scratch_addr[kStaticMaxDevices];
}  // namespace cfx

extern "C" int cfx_strict_forward_static(int device, const float* params, int hidden, int layers,
                                         int num_actions, int num_envs, float* state,
                                         const cfx_forward_io* io, const uint64_t* step_ctr,
                                         void* stream) {
    using namespace cfx;
    CFX_REQUIRE(params && state && io, "cfx_strict_forward_static: NULL argument");
    CFX_REQUIRE(io->records && io->actions, "cfx_strict_forward_static: records/actions is NULL");
    // same rule as cfx_policy_forward; the encoder reads the tail floats of a record as words
    CFX_REQUIRE(((uintptr_t)io->records & 15) == 0,
                "cfx_strict_forward_static: records not 16-byte aligned");
    int ndev = 0;
    CFX_CUDA(cudaGetDeviceCount(&ndev));
    CFX_REQUIRE(device >= 0 && device < ndev && device < kStaticMaxDevices,
                "cfx_strict_forward_static: device %d of %d", device, ndev);
    CFX_REQUIRE(hidden == kStaticHidden,
                "cfx_strict_forward_static: hidden=%d, the fixed scratch is sized for %d", hidden,
                kStaticHidden);
    CFX_REQUIRE(layers >= 1 && layers <= kStaticMaxLayers,
                "cfx_strict_forward_static: layers=%d exceeds the fixed scratch (max %d)", layers,
                kStaticMaxLayers);
    CFX_REQUIRE(num_actions >= 2 && num_actions <= kMaxActions,
                "cfx_strict_forward_static: num_actions=%d out of [2,%d]", num_actions, kMaxActions);
    CFX_REQUIRE(num_envs > 0 && num_envs % 32 == 0 && num_envs <= kStaticMaxEnvs,
                "cfx_strict_forward_static: num_envs=%d must be a multiple of 32 and at most %d "
                "(size of the fixed scratch)", num_envs, kStaticMaxEnvs);
    CFX_GUARD(device);
    cudaStream_t st = (cudaStream_t)stream;
    if (g_static_scratch_addr[device].load(std::memory_order_acquire) == nullptr) {
        // one-time set-up for this device, with it current: resolve the array's device address.
        // It must not happen while the stream is being captured.
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) cudaGetLastError();
        CFX_REQUIRE(cap == cudaStreamCaptureStatusNone,
                    "cfx_strict_forward_static: the first call on a device does its set-up and "
                    "must come before any stream capture");
        float* addr = nullptr;
        CFX_CUDA(cudaGetSymbolAddress((void**)&addr, g_static_scratch));
        CFX_REQUIRE(addr != nullptr, "cfx_strict_forward_static: no device address for the scratch");
        g_static_scratch_addr[device].store(addr, std::memory_order_release);
    }
    float* base = g_static_scratch_addr[device].load(std::memory_order_acquire);
    const ArenaLayout o = ArenaLayout::make(hidden, layers, num_actions);
    int rc = launch_transpose_gates(params, o, base, hidden, layers, st);
    if (rc) return rc;
    StrictArgs a;
    a.n = num_envs; a.H = hidden; a.L = layers; a.A = num_actions;
    a.params = params;
    a.gates_t = base;
    a.records = io->records;
    a.prev_terminals = io->prev_terminals;
    a.uniforms = io->uniforms;
    a.state = state;
    a.scratch_h[0] = base + kStaticGates;
    a.scratch_h[1] = base + kStaticGates + kStaticLayerBuf;
    a.logits_av = io->logits_av ? io->logits_av : base + kStaticGates + 2 * kStaticLayerBuf;
    a.r_state = io->r_state;
    a.r_state_bf16 = io->r_state_bf16 ? 1 : 0;
    a.env_actions = io->env_actions;
    a.actions = io->actions;
    a.logprobs = io->logprobs;
    a.values = io->values;
    a.seed = io->seed;
    a.env_offset = io->env_offset;
    a.step_ctr = reinterpret_cast<unsigned long long*>(const_cast<uint64_t*>(step_ctr));   // read only: no bump
    return strict_forward(a, st, nullptr);
}
