// Launchers of the strict-fp32 kernels and of the stand-alone stages.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "cfx_common.cuh"

namespace cfx {

struct StrictArgs {
    int n, H, L, A;
    int game = 0;           // CFX_GAME_FULL or CFX_GAME_CLASSIC (148-byte records, gather encoder)
    const float* params;    // fp32 arena
    const float* gates_t;   // what launch_transpose_gates writes
    const uint8_t* records;
    const float* prev_terminals;
    const float* uniforms;
    float* state;           // [L][n][H]
    float* scratch_h[2];    // n H activations each, 16-byte aligned
    float* logits_av;       // [n][A+1]
    float* r_state;
    int r_state_bf16 = 0;   // r_state holds bf16 instead of fp32
    float* env_actions;
    int32_t* actions;
    float* logprobs;
    float* values;
    uint64_t seed, env_offset;
    unsigned long long* step_ctr;   // {Philox offset, blocks finished (bump_step)}
    int bump_step = 0;      // raise the offset after the forward
    int weights_ready = 0;  // nothing queued on the stream writes params or gates_t
};

// what the rules choose for n envs: envs a lane of the layers (0: one sum a gate), three stages or two where that is 4; envs a lane
// of the encoder (0: one sum) and its groups of four units
void strict_tiles(int n, int H, int* layer, int* deep, int* encoder, int* groups);
int strict_forward(const StrictArgs& a, cudaStream_t st, int* launches);
int launch_expand(const uint8_t* rec, float* out, int n, cudaStream_t st);
int launch_classic_expand(const uint8_t* rec, float* out, int n, cudaStream_t st);
int launch_done_to_terminals(const int8_t* done, float* out, int n, cudaStream_t st);
int launch_sample(const float* logits, int ld, int A, const float* u, uint64_t seed,
                  uint64_t env_offset, unsigned long long* step_ctr, int bump, int n,
                  float* env_actions, int32_t* actions, float* logprobs, float* values,
                  cudaStream_t st, int early = 0);
// logits by themselves: [n][ld] and a uniform an env -> action and log-probability
int launch_sample_logits(const float* logits, int ld, int A, const float* u, int n, int32_t* actions, float* logprobs,
                         cudaStream_t st);
int launch_uniforms(uint64_t seed, uint64_t env_offset, uint64_t step, int n, float* u, cudaStream_t st);
// copies `bytes` (a multiple of 16) from page-locked host memory, both 16-byte aligned
int launch_fetch(const void* host, void* dst, size_t bytes, cudaStream_t st);
int launch_bump(unsigned long long* ctr, cudaStream_t st);
// The gate matrices as the layers read them, and whether W_enc has values that are not finite, strict_gate_floats(H, L) in all
constexpr int kOddWords = 64;
constexpr size_t strict_gate_floats(int H, int L) { return (size_t)L * 3 * H * H + kOddWords; }
int launch_transpose_gates(const float* params, const ArenaLayout& o, float* Wt, int H, int L, cudaStream_t st);
// counts the batches' reciprocals that are not 1.0f / d (see k_selftest_reciprocals); waits for the device
int selftest_reciprocals(uint32_t first, uint32_t last, uint32_t far, uint64_t* differing);
int launch_init_uniform(float* w, int count, float bound, uint64_t seed, int subseq, cudaStream_t st);

}  // namespace cfx
