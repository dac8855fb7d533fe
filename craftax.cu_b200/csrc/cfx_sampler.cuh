// Device-side categorical sampler and Philox uniform of the policy head.
#pragma once
#include <curand_kernel.h>
#include <cstdint>

namespace cfx {

// One uniform in (0, 1] for (seed, env, step): the same cuRAND device calls the
// reference issues in k_value_sample (craftax_full.cu:9733-9736).
__device__ __forceinline__ float philox_uniform(uint64_t seed, uint64_t env, uint64_t step) {
    curandStatePhilox4_32_10_t st;
    curand_init(seed ^ 0xA5A5A5A5A5A5A5A5ULL, env, step, &st);
    return curand_uniform(&st);
}

// Softmax-CDF sample with one uniform.  Operation order follows
// cf_nn_sample_action (craftax_full.cu:9147-9165): running max, p = expf(l - m)
// summed in ascending action order, first action whose running sum reaches
// u * total (default A - 1), logprob = l - m - logf(total).  A is a template
// parameter so that p[] stays in registers.
// draw_action: p[] comes in as the exponentials.  The running sums replace them, and as they never fall, the action is the
// number of those that the target is beyond; `at(a, beyond)` is told of every action but the last.
template <int A, typename F>
__device__ __forceinline__ int draw_action(float (&p)[A], float u, float* total, F&& at) {
    float sum = 0.0f;
#pragma unroll
    for (int a = 0; a < A; a++) {
        sum += p[a];
        p[a] = sum;
    }
    const float target = u * sum;
    int action = 0;
#pragma unroll
    for (int a = 0; a < A - 1; a++) {
        const bool beyond = !(target <= p[a]);
        action += beyond ? 1 : 0;
        at(a, beyond);
    }
    *total = sum;
    return action;
}
template <int A>
__device__ __forceinline__ int sample_action(const float (&logits)[A], float u, float* logprob) {
    float m = logits[0];
#pragma unroll
    for (int a = 1; a < A; a++) m = fmaxf(m, logits[a]);
    float p[A];
#pragma unroll
    for (int a = 0; a < A; a++) p[a] = expf(logits[a] - m);
    float la = logits[0], total;
    const int action = draw_action<A>(p, u, &total, [&](int a, bool beyond) { la = beyond ? logits[a + 1] : la; });
    *logprob = la - m - logf(total);
    return action;
}

}  // namespace cfx
