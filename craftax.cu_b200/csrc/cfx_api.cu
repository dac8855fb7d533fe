// C-ABI layer: the policy handle and every extern "C" entry point of cfx.h.
#include <cstdarg>
#include <cstdlib>
#include <cmath>
#include <new>

#include "cfx_common.cuh"
#include "cfx_fused.h"
#include "cfx_strict.h"
#include "cfx_tmap.h"

namespace cfx {

static thread_local char g_err[512] = "";

void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}

int cuda_fail(cudaError_t e, const char* what, const char* file, int line) {
    set_error("CUDA error %d (%s) at %s:%d: %s", (int)e, cudaGetErrorString(e), file, line, what);
    return CFX_ERR_CUDA;
}

unsigned long long current_context_id() {
    typedef CUresult (*PFN_id)(CUcontext, unsigned long long*);
    static const PFN_id get = (PFN_id)driver_entry("cuCtxGetId");
    unsigned long long id = 0;
    return get != nullptr && get(nullptr, &id) == CUDA_SUCCESS ? id : 0ull;
}

}  // namespace cfx

using namespace cfx;

constexpr int kHostSlicesMax = 8;
constexpr size_t kHostSliceEnvs = 32768;   // a slice of the pipelined host-buffer forward for this many envs, from two on
constexpr size_t kHostSmallEnvs = 8192;    // batches whose per-env arrays the kernel reads and writes in host memory

// The handle: role of CuPolicy (craftax_full.cu:11758-11796).
struct cfx_policy {
    int device = 0;
    int n = 0, H = 0, L = 0, A = 0;
    int game = CFX_GAME_FULL, obs = kObs, rec_bytes = kRec;
    int precision = CFX_PREC_FP32;
    size_t param_count = 0;
    float* params = nullptr;        // fp32 arena (device)
    float* gates_t = nullptr;       // strict path: transposed gate matrices
    float* state = nullptr;         // [L][n][H]
    float* scratch_h[2] = {nullptr, nullptr};  // fp32 mode: layer ping-pong
    float* logits_scratch = nullptr;           // [n][A+1] when the caller passes none
    unsigned long long* step_ctr = nullptr;   // {step counter, finished blocks of the fp32 sampler}
    cudaStream_t stream = nullptr;
    FusedPlan* fused = nullptr;
    int last_launches = 0;
    // device staging of cfx_policy_forward_host
    uint8_t* st_records = nullptr;
    float* st_terminals = nullptr;
    float* st_uniforms = nullptr;
    float* st_env_actions = nullptr;
    int32_t* st_actions = nullptr;
    float* st_logprobs = nullptr;
    float* st_values = nullptr;
    float* st_logits = nullptr;
    float* st_r_state = nullptr;
    // cfx_policy_forward_host: streams of the pipelined upload and read-back, events per slice; page-locked memory for
    // what a small batch's kernel reads and writes in place
    cudaStream_t copy_stream = nullptr, out_stream = nullptr;
    cudaEvent_t slice_ready[kHostSlicesMax] = {}, slice_done[kHostSlicesMax] = {};
    cudaEvent_t host_fence = nullptr;
    uint8_t* host_io = nullptr;
};

static void free_dev(void* p) {
    if (p) cudaFree(p);
}

static int policy_refresh_mirrors(cfx_policy* p, cudaStream_t st) {
    if (p->precision != CFX_PREC_FP32) return fused_refresh(p->fused, p->params, st);
    const ArenaLayout o = ArenaLayout::make(p->H, p->L, p->A, p->obs);
    return launch_transpose_gates(p->params, o, p->gates_t, p->H, p->L, st);
}

// What only the fp32 mode needs: the transposed gate matrices, two activation buffers [H][n] and room for the logits.
static int policy_ensure_fp32(cfx_policy* p) {
    if (!p->gates_t) CFX_CUDA(cudaMalloc((void**)&p->gates_t, strict_gate_floats(p->H, p->L) * sizeof(float)));
    for (int i = 0; i < 2; i++)
        if (!p->scratch_h[i]) CFX_CUDA(cudaMalloc((void**)&p->scratch_h[i], (size_t)p->H * p->n * sizeof(float)));
    if (!p->logits_scratch)
        CFX_CUDA(cudaMalloc((void**)&p->logits_scratch, (size_t)p->n * (p->A + 1) * sizeof(float)));
    return CFX_OK;
}

static int require_fused(const cfx_policy* p, int precision) {
    if (fused_supported(p->H, p->L, p->A, precision, p->game)) return CFX_OK;
    set_error("precision %d is not built for hidden=%d layers=%d actions=%d", precision, p->H, p->L, p->A);
    return CFX_ERR_UNSUPPORTED;
}

extern "C" {

const char* cfx_last_error(void) { return g_err; }
const char* cfx_version(void) { return "cfx-b200 0.1 (sm_100a)"; }

size_t cfx_param_count(int hidden, int layers, int num_actions) {
    if (hidden <= 0 || layers <= 0 || num_actions <= 0) return 0;
    return ArenaLayout::make(hidden, layers, num_actions).count;
}

static int policy_create(cfx_policy** out, int device, int num_envs, int hidden, int layers,
                         int num_actions, int precision, int game);

int cfx_policy_create(cfx_policy** out, int device, int num_envs, int hidden, int layers,
                      int num_actions, int precision) {
    return policy_create(out, device, num_envs, hidden, layers, num_actions, precision, CFX_GAME_FULL);
}

int cfx_policy_create_classic(cfx_policy** out, int device, int num_envs, int hidden, int layers,
                              int num_actions, int precision) {
    return policy_create(out, device, num_envs, hidden, layers, num_actions, precision, CFX_GAME_CLASSIC);
}

size_t cfx_classic_param_count(int hidden, int layers, int num_actions) {
    if (hidden <= 0 || layers <= 0 || num_actions <= 0) return 0;
    return ArenaLayout::make(hidden, layers, num_actions, kClassicObs).count;
}

int cfx_classic_expand_obs(int device, const uint8_t* records, float* out, int num_envs, void* stream) {
    CFX_REQUIRE(records && out && num_envs > 0, "cfx_classic_expand_obs: bad arguments");
    CFX_GUARD(device);
    return launch_classic_expand(records, out, num_envs, (cudaStream_t)stream);
}

int cfx_classic_done_to_terminals(int device, const int8_t* done, float* out, int num_envs, void* stream) {
    CFX_REQUIRE(done && out && num_envs > 0, "cfx_classic_done_to_terminals: bad arguments");
    CFX_GUARD(device);
    return launch_done_to_terminals(done, out, num_envs, (cudaStream_t)stream);
}

static int policy_create(cfx_policy** out, int device, int num_envs, int hidden, int layers,
                         int num_actions, int precision, int game) {
    CFX_REQUIRE(out != nullptr, "cfx_policy_create: out is NULL");
    *out = nullptr;
    CFX_REQUIRE(num_envs > 0 && num_envs % 32 == 0,
                "cfx_policy_create: num_envs=%d must be a positive multiple of 32", num_envs);
    CFX_REQUIRE(hidden >= 32 && hidden <= kMaxHidden && hidden % 32 == 0,
                "cfx_policy_create: hidden=%d must be a multiple of 32 in [32,%d]", hidden, kMaxHidden);
    CFX_REQUIRE(layers >= 1 && layers <= 8, "cfx_policy_create: layers=%d out of [1,8]", layers);
    CFX_REQUIRE(num_actions >= 2 && num_actions <= kMaxActions,
                "cfx_policy_create: num_actions=%d out of [2,%d]", num_actions, kMaxActions);
    CFX_REQUIRE(precision >= CFX_PREC_FP32 && precision <= CFX_PREC_TF32,
                "cfx_policy_create: unknown precision %d", precision);
    int ndev = 0;
    CFX_CUDA(cudaGetDeviceCount(&ndev));
    CFX_REQUIRE(device >= 0 && device < ndev, "cfx_policy_create: device %d of %d", device, ndev);
    CFX_GUARD(device);
    cfx_policy* p = new (std::nothrow) cfx_policy();
    CFX_REQUIRE(p != nullptr, "cfx_policy_create: out of host memory");
    p->device = device;
    p->n = num_envs;
    p->H = hidden;
    p->L = layers;
    p->A = num_actions;
    p->precision = precision;
    p->game = game;
    p->obs = game == CFX_GAME_CLASSIC ? kClassicObs : kObs;
    p->rec_bytes = game == CFX_GAME_CLASSIC ? kClassicRec : kRec;
    p->param_count = ArenaLayout::make(hidden, layers, num_actions, p->obs).count;
    const size_t hn = (size_t)hidden * num_envs;
    int rc = CFX_OK;
    auto fail = [&](int code) {
        cfx_policy_destroy(p);
        return code;
    };
#define CFX_TRY_ALLOC(ptr, bytes)                                                    \
    do {                                                                             \
        cudaError_t _e = cudaMalloc((void**)&(ptr), (bytes));                        \
        if (_e != cudaSuccess) return fail(cuda_fail(_e, "cudaMalloc " #ptr, __FILE__, __LINE__)); \
    } while (0)
    CFX_TRY_ALLOC(p->params, p->param_count * sizeof(float));
    CFX_TRY_ALLOC(p->state, (size_t)layers * hn * sizeof(float));
    CFX_TRY_ALLOC(p->step_ctr, 2 * sizeof(unsigned long long));
#undef CFX_TRY_ALLOC
    cudaError_t e = cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) return fail(cuda_fail(e, "cudaStreamCreateWithFlags", __FILE__, __LINE__));
    e = cudaMemsetAsync(p->params, 0, p->param_count * sizeof(float), p->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(p->state, 0, (size_t)layers * hn * sizeof(float), p->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(p->step_ctr, 0, 2 * sizeof(unsigned long long), p->stream);
    if (e != cudaSuccess) return fail(cuda_fail(e, "cudaMemsetAsync", __FILE__, __LINE__));
    if (precision == CFX_PREC_FP32) rc = policy_ensure_fp32(p);
    else if ((rc = require_fused(p, precision)) == CFX_OK)
        rc = fused_create(&p->fused, device, num_envs, hidden, layers, num_actions, precision, p->state, game);
    if (rc) return fail(rc);
    rc = policy_refresh_mirrors(p, p->stream);
    if (rc) return fail(rc);
    e = cudaStreamSynchronize(p->stream);
    if (e != cudaSuccess) return fail(cuda_fail(e, "cudaStreamSynchronize", __FILE__, __LINE__));
    *out = p;
    return CFX_OK;
}

int cfx_policy_destroy(cfx_policy* p) {
    if (!p) return CFX_OK;
    DeviceGuard g(p->device);   // best effort: the handle is released whatever happens
    if (p->stream) cudaStreamSynchronize(p->stream);
    if (p->fused) fused_destroy(p->fused);
    free_dev(p->params);
    free_dev(p->gates_t);
    free_dev(p->state);
    free_dev(p->scratch_h[0]);
    free_dev(p->scratch_h[1]);
    free_dev(p->logits_scratch);
    free_dev(p->step_ctr);
    free_dev(p->st_records);
    free_dev(p->st_terminals);
    free_dev(p->st_uniforms);
    free_dev(p->st_env_actions);
    free_dev(p->st_actions);
    free_dev(p->st_logprobs);
    free_dev(p->st_values);
    free_dev(p->st_logits);
    free_dev(p->st_r_state);
    for (int i = 0; i < kHostSlicesMax; i++) {
        if (p->slice_ready[i]) cudaEventDestroy(p->slice_ready[i]);
        if (p->slice_done[i]) cudaEventDestroy(p->slice_done[i]);
    }
    if (p->host_fence) cudaEventDestroy(p->host_fence);
    if (p->copy_stream) cudaStreamDestroy(p->copy_stream);
    if (p->out_stream) cudaStreamDestroy(p->out_stream);
    if (p->host_io) cudaFreeHost(p->host_io);
    if (p->stream) cudaStreamDestroy(p->stream);
    delete p;
    return CFX_OK;
}

int cfx_policy_set_weights(cfx_policy* p, const float* arena, size_t count, int on_device) {
    CFX_REQUIRE(p && arena, "cfx_policy_set_weights: NULL argument");
    CFX_REQUIRE(count == p->param_count, "cfx_policy_set_weights: count %zu != %zu", count,
                p->param_count);
    CFX_GUARD(p->device);
    CFX_CUDA(cudaMemcpyAsync(p->params, arena, count * sizeof(float),
                             on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice,
                             p->stream));
    int rc = policy_refresh_mirrors(p, p->stream);
    if (rc) return rc;
    CFX_CUDA(cudaStreamSynchronize(p->stream));
    return CFX_OK;
}

int cfx_policy_get_weights(cfx_policy* p, float* host_arena, size_t count) {
    CFX_REQUIRE(p && host_arena, "cfx_policy_get_weights: NULL argument");
    CFX_REQUIRE(count == p->param_count, "cfx_policy_get_weights: count %zu != %zu", count,
                p->param_count);
    CFX_GUARD(p->device);
    CFX_CUDA(cudaMemcpyAsync(host_arena, p->params, count * sizeof(float), cudaMemcpyDeviceToHost,
                             p->stream));
    CFX_CUDA(cudaStreamSynchronize(p->stream));
    return CFX_OK;
}

int cfx_policy_init_weights(cfx_policy* p, uint64_t seed) {
    CFX_REQUIRE(p, "cfx_policy_init_weights: NULL handle");
    CFX_GUARD(p->device);
    const ArenaLayout o = ArenaLayout::make(p->H, p->L, p->A, p->obs);
    const float be = 1.0f / sqrtf((float)p->obs), bh = 1.0f / sqrtf((float)p->H);
    const struct { size_t off; size_t count; float bound; } segs[7] = {
        {o.w_enc, (size_t)p->obs * p->H, be}, {o.b_enc, (size_t)p->H, be},
        {o.w_gru, (size_t)p->L * 3 * p->H * p->H, bh}, {o.w_a, (size_t)p->A * p->H, bh},
        {o.b_a, (size_t)p->A, bh}, {o.w_v, (size_t)p->H, bh}, {o.b_v, 1, bh}};
    for (int s = 0; s < 7; s++) {
        int rc = launch_init_uniform(p->params + segs[s].off, (int)segs[s].count, segs[s].bound,
                                     seed, s, p->stream);
        if (rc) return rc;
    }
    int rc = policy_refresh_mirrors(p, p->stream);
    if (rc) return rc;
    CFX_CUDA(cudaStreamSynchronize(p->stream));
    return CFX_OK;
}

}  // extern "C"

// ------------------------------------------------------------------ checkpoint
static const uint32_t kCkptMagic = 0x31574643u;  // "CFW1", craftax_full.cu:12243

extern "C" {

int cfx_policy_save_cfw1(cfx_policy* p, const char* path) {
    CFX_REQUIRE(p && path, "cfx_policy_save_cfw1: NULL argument");
    float* h = (float*)malloc(p->param_count * sizeof(float));
    CFX_REQUIRE(h != nullptr, "cfx_policy_save_cfw1: out of host memory");
    int rc = cfx_policy_get_weights(p, h, p->param_count);
    if (rc) { free(h); return rc; }
    FILE* f = fopen(path, "wb");
    if (!f) {
        free(h);
        set_error("cfx_policy_save_cfw1: cannot write %s", path);
        return CFX_ERR_IO;
    }
    const uint32_t hdr[4] = {kCkptMagic, (uint32_t)p->H, (uint32_t)p->L, (uint32_t)p->param_count};
    bool ok = fwrite(hdr, sizeof(hdr), 1, f) == 1 &&
              fwrite(h, sizeof(float), p->param_count, f) == p->param_count;
    ok = (fclose(f) == 0) && ok;
    free(h);
    if (!ok) {
        set_error("cfx_policy_save_cfw1: short write to %s", path);
        return CFX_ERR_IO;
    }
    return CFX_OK;
}

int cfx_policy_load_cfw1(cfx_policy* p, const char* path) {
    CFX_REQUIRE(p && path, "cfx_policy_load_cfw1: NULL argument");
    FILE* f = fopen(path, "rb");
    if (!f) {
        set_error("cfx_policy_load_cfw1: cannot read %s", path);
        return CFX_ERR_IO;
    }
    uint32_t hdr[4];
    if (fread(hdr, sizeof(hdr), 1, f) != 1 || hdr[0] != kCkptMagic || hdr[1] != (uint32_t)p->H ||
        hdr[2] != (uint32_t)p->L || hdr[3] != (uint32_t)p->param_count) {
        fclose(f);
        set_error("cfx_policy_load_cfw1: %s: bad header (want h%dx%d, %zu params)", path, p->H,
                  p->L, p->param_count);
        return CFX_ERR_IO;
    }
    float* h = (float*)malloc(p->param_count * sizeof(float));
    if (!h) {
        fclose(f);
        set_error("cfx_policy_load_cfw1: out of host memory");
        return CFX_ERR_INVALID;
    }
    size_t got = fread(h, sizeof(float), p->param_count, f);
    fclose(f);
    if (got != p->param_count) {
        free(h);
        set_error("cfx_policy_load_cfw1: %s: truncated", path);
        return CFX_ERR_IO;
    }
    int rc = cfx_policy_set_weights(p, h, p->param_count, 0);
    free(h);
    return rc;
}

int cfx_policy_set_precision(cfx_policy* p, int precision) {
    CFX_REQUIRE(p, "cfx_policy_set_precision: NULL handle");
    CFX_REQUIRE(precision >= CFX_PREC_FP32 && precision <= CFX_PREC_TF32,
                "cfx_policy_set_precision: unknown precision %d", precision);
    if (precision == p->precision) return CFX_OK;
    CFX_GUARD(p->device);
    CFX_CUDA(cudaStreamSynchronize(p->stream));
    int rc;
    if (precision != CFX_PREC_FP32 && (rc = require_fused(p, precision))) return rc;
    // What the handle uses stays as it is until the new operands are complete: a refused switch leaves it untouched (a
    // captured graph holds its pointers), and no forward reads operands that are still being written (the
    // kernels read them before they wait for the work in front of them).
    FusedPlan* plan = nullptr;
    if (precision == CFX_PREC_FP32) {
        if ((rc = policy_ensure_fp32(p))) return rc;
        const ArenaLayout o = ArenaLayout::make(p->H, p->L, p->A, p->obs);
        rc = launch_transpose_gates(p->params, o, p->gates_t, p->H, p->L, p->stream);
    } else {
        if ((rc = fused_create(&plan, p->device, p->n, p->H, p->L, p->A, precision, p->state, p->game))) return rc;
        rc = fused_refresh(plan, p->params, p->stream);
    }
    if (rc == CFX_OK) {
        const cudaError_t e = cudaStreamSynchronize(p->stream);
        if (e != cudaSuccess) rc = cuda_fail(e, "cudaStreamSynchronize", __FILE__, __LINE__);
    }
    if (rc) {
        fused_destroy(plan);
        return rc;
    }
    fused_destroy(p->fused);
    p->fused = plan;
    p->precision = precision;
    return CFX_OK;
}

int cfx_policy_get_precision(const cfx_policy* p) { return p ? p->precision : -1; }

float* cfx_policy_state(cfx_policy* p) { return p ? p->state : nullptr; }

int cfx_policy_reset_state(cfx_policy* p, void* stream) {
    CFX_REQUIRE(p, "cfx_policy_reset_state: NULL handle");
    CFX_GUARD(p->device);
    cudaStream_t st = stream ? (cudaStream_t)stream : p->stream;
    CFX_CUDA(cudaMemsetAsync(p->state, 0, (size_t)p->L * p->n * p->H * sizeof(float), st));
    return CFX_OK;
}

int cfx_policy_set_step(cfx_policy* p, uint64_t step, void* stream) {
    CFX_REQUIRE(p, "cfx_policy_set_step: NULL handle");
    CFX_GUARD(p->device);
    cudaStream_t st = stream ? (cudaStream_t)stream : p->stream;
    unsigned long long v = step;
    CFX_CUDA(cudaMemcpyAsync(p->step_ctr, &v, sizeof(v), cudaMemcpyHostToDevice, st));
    CFX_CUDA(cudaStreamSynchronize(st));
    return CFX_OK;
}

int cfx_policy_get_step(cfx_policy* p, uint64_t* step) {
    CFX_REQUIRE(p && step, "cfx_policy_get_step: NULL argument");
    CFX_GUARD(p->device);
    unsigned long long v = 0;
    CFX_CUDA(cudaMemcpyAsync(&v, p->step_ctr, sizeof(v), cudaMemcpyDeviceToHost, p->stream));
    CFX_CUDA(cudaStreamSynchronize(p->stream));
    *step = v;
    return CFX_OK;
}

int cfx_policy_bump_step(cfx_policy* p, void* stream) {
    CFX_REQUIRE(p, "cfx_policy_bump_step: NULL handle");
    CFX_GUARD(p->device);
    return launch_bump(p->step_ctr, stream ? (cudaStream_t)stream : p->stream);
}

void* cfx_policy_stream(cfx_policy* p) { return p ? (void*)p->stream : nullptr; }
int cfx_policy_last_launches(const cfx_policy* p) { return p ? p->last_launches : 0; }

// ------------------------------------------------------------------ forward
// One forward over the 128-env tiles [tile_begin, tile_end) of the batch (tile_end = 0: all;
// slices are a fused-kernel feature, used by the pipelined host-buffer forward).
static int forward_range(cfx_policy* p, const cfx_forward_io* io, void* stream, int tile_begin, int tile_end) {
    CFX_REQUIRE(p && io, "cfx_policy_forward: NULL argument");
    CFX_REQUIRE(io->records != nullptr, "cfx_policy_forward: records is NULL");
    CFX_REQUIRE(((uintptr_t)io->records & 15) == 0, "cfx_policy_forward: records not 16-byte aligned");
    CFX_REQUIRE(io->actions != nullptr, "cfx_policy_forward: actions is NULL");
    CFX_GUARD(p->device);
    cudaStream_t st = stream ? (cudaStream_t)stream : p->stream;
    int launches = 0, rc;
    if (p->precision == CFX_PREC_FP32) {
        StrictArgs a;
        a.n = p->n; a.H = p->H; a.L = p->L; a.A = p->A;
        a.game = p->game;
        a.params = p->params;
        a.gates_t = p->gates_t;
        a.records = io->records;
        a.prev_terminals = io->prev_terminals;
        a.uniforms = io->uniforms;
        a.state = p->state;
        a.scratch_h[0] = p->scratch_h[0];
        a.scratch_h[1] = p->scratch_h[1];
        a.logits_av = io->logits_av ? io->logits_av : p->logits_scratch;
        a.r_state = io->r_state;
        a.r_state_bf16 = io->r_state_bf16 ? 1 : 0;
        a.env_actions = io->env_actions;
        a.actions = io->actions;
        a.logprobs = io->logprobs;
        a.values = io->values;
        a.seed = io->seed;
        a.env_offset = io->env_offset;
        a.step_ctr = p->step_ctr;
        a.bump_step = io->bump_step ? 1 : 0;
        a.weights_ready = 1;
        rc = strict_forward(a, st, &launches);
    } else {
        CFX_REQUIRE(p->fused != nullptr, "cfx_policy_forward: fused plan missing");
        FusedArgs a;
        a.records = io->records;
        a.prev_terminals = io->prev_terminals;
        a.uniforms = io->uniforms;
        a.state = p->state;
        a.env_actions = io->env_actions;
        a.actions = io->actions;
        a.logprobs = io->logprobs;
        a.values = io->values;
        a.logits_av = io->logits_av;
        a.r_state = io->r_state;
        a.r_state_bf16 = io->r_state_bf16 ? 1 : 0;
        a.seed = io->seed;
        a.env_offset = io->env_offset;
        a.step_ctr = p->step_ctr;
        a.bump_step = io->bump_step ? 1 : 0;   // folded into the kernel: no extra launch
        a.tile_begin = tile_begin;
        a.tile_end = tile_end;
        rc = fused_forward(p->fused, a, st, &launches);
    }
    if (rc) return rc;
    p->last_launches = launches;
    return CFX_OK;
}

int cfx_policy_forward(cfx_policy* p, const cfx_forward_io* io, void* stream) {
    return forward_range(p, io, stream, 0, 0);
}

}  // extern "C"

static int check_status(cfx_policy* p);

extern "C" int cfx_policy_check(cfx_policy* p, void* stream) {
    CFX_REQUIRE(p, "cfx_policy_check: NULL handle");
    CFX_GUARD(p->device);
    CFX_CUDA(cudaStreamSynchronize(stream ? (cudaStream_t)stream : p->stream));
    return check_status(p);
}

extern "C" int cfx_selftest_wait_timeout(int device, unsigned limit_ms) {
    CFX_REQUIRE(limit_ms >= 1 && limit_ms <= 1000, "cfx_selftest_wait_timeout: limit_ms=%u out of [1,1000]", limit_ms);
    CFX_GUARD(device);
    unsigned status = 0;
    int rc = fused_selftest_wait_timeout(limit_ms, &status);
    if (rc) return rc;
    if (status == 0) {
        set_error("self-test: the bounded wait did not report a timeout");
        return CFX_ERR_CUDA;
    }
    set_error("device-side wait timed out: site %u, block %u (self-test)", status & 0xFF, status >> 8);
    return CFX_ERR_DEVICE_TIMEOUT;
}

extern "C" int cfx_selftest_reciprocals(int device, uint32_t first, uint32_t last, uint32_t far, uint64_t* differing) {
    CFX_REQUIRE(differing, "cfx_selftest_reciprocals: NULL argument");
    CFX_REQUIRE(first >= 0x3F800000u && first <= last && last <= 0x7FFFFFFFu, "cfx_selftest_reciprocals: bits %x .. %x", first, last);
    CFX_GUARD(device);
    return selftest_reciprocals(first, last, far, differing);
}

extern "C" int cfx_selftest_strict_tiles(int num_envs, int hidden, int32_t* tiles) {
    CFX_REQUIRE(tiles && num_envs > 0 && num_envs % 32 == 0 && hidden > 0 && hidden % 32 == 0 && hidden <= kMaxHidden,
                "cfx_selftest_strict_tiles: %d envs, hidden %d", num_envs, hidden);
    strict_tiles(num_envs, hidden, tiles, tiles + 1, tiles + 2, tiles + 3);
    return CFX_OK;
}

// ------------------------------------------------------------------ host-buffer forward
template <typename T>
static int ensure_staging(T** slot, size_t count) {
    if (*slot) return CFX_OK;
    CFX_CUDA(cudaMalloc((void**)slot, count * sizeof(T)));
    return CFX_OK;
}

static int check_status(cfx_policy* p) {
    const unsigned status = p->fused ? fused_take_status(p->fused) : 0u;
    if (status == 0) return CFX_OK;
    set_error("device-side wait timed out: site %u, block %u", status & 0xFF, status >> 8);
    return CFX_ERR_DEVICE_TIMEOUT;
}

static bool page_locked(const void* host) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost;
}

// The device's address of [host, host + bytes) where all of it lies in one piece of page-locked memory (allocated, or
// registered as a whole), or NULL: a kernel that went past the end of such a piece would fault.
static void* device_address(const void* host, size_t bytes) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    if (a.type != cudaMemoryTypeHost || a.devicePointer == nullptr) return nullptr;
    typedef CUresult (*PFN_attribute)(void*, CUpointer_attribute, CUdeviceptr);
    static const PFN_attribute attribute = (PFN_attribute)driver_entry("cuPointerGetAttribute");
    const uintptr_t at = (uintptr_t)a.devicePointer;
    CUdeviceptr start = 0;
    size_t size = 0;
    if (attribute == nullptr || attribute(&start, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, (CUdeviceptr)at) != CUDA_SUCCESS ||
        attribute(&size, CU_POINTER_ATTRIBUTE_RANGE_SIZE, (CUdeviceptr)at) != CUDA_SUCCESS)
        return nullptr;
    return at >= start && at - start <= size && bytes <= size - (at - start) ? a.devicePointer : nullptr;
}

// Small batches, fused kernel: what such a step costs is calls and round trips, not bytes.  Flags, uniforms and the four
// per-env outputs are read and written by the kernel in page-locked host memory of the handle (a few KB, copied
// from and to the caller's arrays here).  The smallest batches' records are fetched by a kernel, which saves the
// hand-over between a copy engine and the SMs, and their logits are written in place: to the caller's array where it
// is page-locked, else by way of the handle's.  Beyond, a copy moves them faster than the SMs do over PCIe.
// us a call, with a copy for each array and for the status word before -> now: 32 envs 82 -> 42, 1,024 envs 108 -> 68,
// 4,096 envs 178 -> 150 (512 envs: 58 with the records fetched by the kernel, 55 copied).
constexpr size_t kHostFetchEnvs = 256, kHostLogitsEnvs = 2048, kHostLogitsCopyEnvs = 256;
static int forward_host_small(cfx_policy* p, const cfx_forward_io* h, cfx_forward_io* d) {
    cudaStream_t st = p->stream;
    const size_t n = (size_t)p->n, row = (size_t)(p->A + 1) * 4;
    if (!p->host_io)
        CFX_CUDA(cudaHostAlloc((void**)&p->host_io, 6 * n * 4 + (n <= kHostLogitsCopyEnvs ? n * row : 0),
                               cudaHostAllocPortable | cudaHostAllocMapped));
    auto part = [&](int i) { return p->host_io + (size_t)i * n * 4; };   // n is a multiple of 32: 128-byte aligned
    auto in = [&](const float* src, int i) -> const float* {
        if (!src) return nullptr;
        memcpy(part(i), src, n * 4);
        return (const float*)part(i);
    };
    d->prev_terminals = in(h->prev_terminals, 0);
    d->uniforms = in(h->uniforms, 1);
    d->env_actions = h->env_actions ? (float*)part(2) : nullptr;
    d->actions = (int32_t*)part(3);
    d->logprobs = h->logprobs ? (float*)part(4) : nullptr;
    d->values = h->values ? (float*)part(5) : nullptr;
    void* logits = h->logits_av && n <= kHostLogitsEnvs ? device_address(h->logits_av, n * row) : nullptr;
    if (logits && ((uintptr_t)logits & 15) != 0) logits = nullptr;
    const bool staged = h->logits_av && !logits && n <= kHostLogitsCopyEnvs;
    if (staged) logits = part(6);
    if (logits) d->logits_av = (float*)logits;
    const size_t bytes = n * (size_t)p->rec_bytes;
    const void* rec = n <= kHostFetchEnvs ? device_address(h->records, bytes) : nullptr;
    int rc;
    const bool fetch = rec && ((uintptr_t)rec & 15) == 0;
    if (fetch) {
        if ((rc = launch_fetch(rec, p->st_records, bytes, st))) return rc;
    } else {
        CFX_CUDA(cudaMemcpyAsync(p->st_records, h->records, bytes, cudaMemcpyHostToDevice, st));
    }
    if ((rc = cfx_policy_forward(p, d, st))) return rc;
    p->last_launches += fetch ? 1 : 0;
    if (h->logits_av && !logits)
        CFX_CUDA(cudaMemcpyAsync(h->logits_av, p->st_logits, n * row, cudaMemcpyDeviceToHost, st));
    if (h->r_state)
        CFX_CUDA(cudaMemcpyAsync(h->r_state, p->st_r_state, (size_t)p->L * n * p->H * (h->r_state_bf16 ? 2 : 4),
                                 cudaMemcpyDeviceToHost, st));
    CFX_CUDA(cudaStreamSynchronize(st));
    if ((rc = check_status(p))) return rc;
    auto out = [&](void* dst, int i, size_t bytes_out) {
        if (dst) memcpy(dst, part(i), bytes_out);
    };
    out(h->env_actions, 2, n * 4);
    out(h->actions, 3, n * 4);
    out(h->logprobs, 4, n * 4);
    out(h->values, 5, n * 4);
    if (staged) out(h->logits_av, 6, n * row);
    return CFX_OK;
}

extern "C" {

int cfx_policy_forward_host(cfx_policy* p, const cfx_forward_io* h) {
    CFX_REQUIRE(p && h, "cfx_policy_forward_host: NULL argument");
    CFX_REQUIRE(h->records && h->actions, "cfx_policy_forward_host: records/actions is NULL");
    CFX_GUARD(p->device);
    cudaStream_t st = p->stream;
    const size_t n = (size_t)p->n;
    const bool fused = p->precision != CFX_PREC_FP32, small = fused && n < kHostSmallEnvs;
    const size_t lav = (size_t)(p->A + 1);
    int rc;
    if ((rc = ensure_staging(&p->st_records, n * (size_t)p->rec_bytes))) return rc;
    if (h->logits_av && (rc = ensure_staging(&p->st_logits, n * lav))) return rc;
    if (h->r_state && (rc = ensure_staging(&p->st_r_state, (size_t)p->L * n * p->H))) return rc;
    cfx_forward_io d = *h;
    d.records = p->st_records;
    d.logits_av = h->logits_av ? p->st_logits : nullptr;
    d.r_state = h->r_state ? p->st_r_state : nullptr;
    if (small) return forward_host_small(p, h, &d);

    if ((rc = ensure_staging(&p->st_actions, n))) return rc;
    if (h->prev_terminals && (rc = ensure_staging(&p->st_terminals, n))) return rc;
    if (h->uniforms && (rc = ensure_staging(&p->st_uniforms, n))) return rc;
    if (h->env_actions && (rc = ensure_staging(&p->st_env_actions, n))) return rc;
    if (h->logprobs && (rc = ensure_staging(&p->st_logprobs, n))) return rc;
    if (h->values && (rc = ensure_staging(&p->st_values, n))) return rc;
    d.prev_terminals = h->prev_terminals ? p->st_terminals : nullptr;
    d.uniforms = h->uniforms ? p->st_uniforms : nullptr;
    d.env_actions = h->env_actions ? p->st_env_actions : nullptr;
    d.actions = p->st_actions;
    d.logprobs = h->logprobs ? p->st_logprobs : nullptr;
    d.values = h->values ? p->st_values : nullptr;
    auto inputs = [&](cudaStream_t s) {
        cudaError_t e = cudaSuccess;
        if (h->prev_terminals)
            e = cudaMemcpyAsync(p->st_terminals, h->prev_terminals, n * sizeof(float), cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess && h->uniforms)
            e = cudaMemcpyAsync(p->st_uniforms, h->uniforms, n * sizeof(float), cudaMemcpyHostToDevice, s);
        return e;
    };
    // the outputs of envs [e0, e1)
    auto outputs = [&](size_t e0, size_t e1, cudaStream_t s) {
        auto one = [&](void* dst, const void* src, size_t words) {
            if (!dst) return cudaSuccess;
            return cudaMemcpyAsync((uint8_t*)dst + e0 * words * 4, (const uint8_t*)src + e0 * words * 4, (e1 - e0) * words * 4,
                                   cudaMemcpyDeviceToHost, s);
        };
        cudaError_t e = one(h->logits_av, p->st_logits, lav);
        if (e == cudaSuccess) e = one(h->actions, p->st_actions, 1);
        if (e == cudaSuccess) e = one(h->env_actions, p->st_env_actions, 1);
        if (e == cudaSuccess) e = one(h->logprobs, p->st_logprobs, 1);
        if (e == cudaSuccess) e = one(h->values, p->st_values, 1);
        return e;
    };
    cudaStream_t last = st;   // the stream whose end is the end of the call
    if (!fused || n < 2 * kHostSliceEnvs) {
        CFX_CUDA(cudaMemcpyAsync(p->st_records, h->records, n * (size_t)p->rec_bytes, cudaMemcpyHostToDevice, st));
        CFX_CUDA(inputs(st));
        rc = cfx_policy_forward(p, &d, st);
        if (rc) return rc;
        CFX_CUDA(outputs(0, n, st));
    } else {
        // The record upload dominates a host-buffer step (996 bytes per env over PCIe against 192 bytes of outputs the other
        // way and ~1.6 ns of kernel time).  The records go up in slices on a stream of their own, the kernel runs slice by
        // slice behind them (a launch takes a tile range) and the outputs of a slice go down on a third stream, so
        // that only the last slice's kernel and outputs are not hidden under the upload.  The slices shrink: a slice's kernel
        // and outputs take a third of its upload, so that each is done when the next, smaller one has arrived.
        // 65,536 envs: 1,533 us with two equal slices and the outputs at the end, 1,357 us now (the upload alone 1,180).
        int slices = (int)(n / kHostSliceEnvs);
        slices = slices > kHostSlicesMax ? kHostSlicesMax : slices;
        if (!p->copy_stream) {
            CFX_CUDA(cudaStreamCreateWithFlags(&p->copy_stream, cudaStreamNonBlocking));
            CFX_CUDA(cudaStreamCreateWithFlags(&p->out_stream, cudaStreamNonBlocking));
            CFX_CUDA(cudaEventCreateWithFlags(&p->host_fence, cudaEventDisableTiming));
            for (int i = 0; i < kHostSlicesMax; i++) {
                CFX_CUDA(cudaEventCreateWithFlags(&p->slice_ready[i], cudaEventDisableTiming));
                CFX_CUDA(cudaEventCreateWithFlags(&p->slice_done[i], cudaEventDisableTiming));
            }
        }
        cudaStream_t cs = p->copy_stream;
        // A copy to pageable memory holds up the host, and with it the uploads behind it: where an output is such memory, all go
        // down at the end (262,144 envs, records page-locked, outputs not: 8,410 us slice by slice, 7,410 so).
        bool locked = true;
        for (const void* dst : {(const void*)h->logits_av, (const void*)h->actions, (const void*)h->env_actions,
                                (const void*)h->logprobs, (const void*)h->values})
            locked = locked && (dst == nullptr || page_locked(dst));
        // the staging buffers may still be read by work queued earlier on the handle's stream
        CFX_CUDA(cudaEventRecord(p->host_fence, st));
        CFX_CUDA(cudaStreamWaitEvent(cs, p->host_fence, 0));
        CFX_CUDA(inputs(cs));
        // what is left after slice k: from the whole batch down to the last slice in equal ratios
        const double end = (double)n / 5 < 16384 ? (double)n / 5 : 16384.0, ratio = pow(end / (double)n, 1.0 / (slices - 1));
        const int tiles = (int)((n + 127) / 128);
        double left = (double)n;
        int launches = 0;
        for (int k = 0, t0 = 0; t0 < tiles; k++) {
            left *= ratio;
            int t1 = k == slices - 1 ? tiles : (int)(((double)n - left) / 128);
            t1 += t1 & 1;   // slices start at even tiles (CTA pairs)
            t1 = t1 < t0 + 2 ? t0 + 2 : t1;
            t1 = t1 > tiles ? tiles : t1;
            const size_t e0 = (size_t)t0 * 128, e1 = (size_t)t1 * 128 < n ? (size_t)t1 * 128 : n;
            CFX_CUDA(cudaMemcpyAsync(p->st_records + e0 * p->rec_bytes, h->records + e0 * p->rec_bytes,
                                     (e1 - e0) * (size_t)p->rec_bytes, cudaMemcpyHostToDevice, cs));
            CFX_CUDA(cudaEventRecord(p->slice_ready[k], cs));
            CFX_CUDA(cudaStreamWaitEvent(st, p->slice_ready[k], 0));
            cfx_forward_io dk = d;
            dk.bump_step = (t1 == tiles) ? h->bump_step : 0;   // the last slice bumps the counter
            rc = forward_range(p, &dk, st, t0, t1);
            if (rc) return rc;
            launches += p->last_launches;
            if (locked) {
                CFX_CUDA(cudaEventRecord(p->slice_done[k], st));
                CFX_CUDA(cudaStreamWaitEvent(p->out_stream, p->slice_done[k], 0));
                CFX_CUDA(outputs(e0, e1, p->out_stream));
            }
            t0 = t1;
        }
        p->last_launches = launches;
        if (locked) last = p->out_stream;
        else CFX_CUDA(outputs(0, n, st));
    }
    if (h->r_state)
        CFX_CUDA(cudaMemcpyAsync(h->r_state, p->st_r_state, (size_t)p->L * n * p->H * (h->r_state_bf16 ? 2 : 4),
                                 cudaMemcpyDeviceToHost, last));
    CFX_CUDA(cudaStreamSynchronize(last));
    return check_status(p);
}

// ------------------------------------------------------------------ stand-alone stages
int cfx_expand_obs(int device, const uint8_t* records, float* features, int n, void* stream) {
    CFX_REQUIRE(records && features && n > 0, "cfx_expand_obs: bad argument");
    // the 51 tail floats of a record are read as 32-bit words
    CFX_REQUIRE(((uintptr_t)records & 3) == 0, "cfx_expand_obs: records not 4-byte aligned");
    CFX_GUARD(device);
    return launch_expand(records, features, n, (cudaStream_t)stream);
}

int cfx_sample_actions(int device, const float* logits, int ld, int num_actions,
                       const float* uniforms, int n, int32_t* actions, float* logprobs,
                       void* stream) {
    CFX_REQUIRE(logits && uniforms && actions && logprobs && n > 0, "cfx_sample_actions: bad argument");
    CFX_REQUIRE(num_actions >= 2 && num_actions <= kMaxActions && ld >= num_actions,
                "cfx_sample_actions: num_actions=%d ld=%d", num_actions, ld);
    CFX_GUARD(device);
    return launch_sample_logits(logits, ld, num_actions, uniforms, n, actions, logprobs, (cudaStream_t)stream);
}

int cfx_philox_uniforms(int device, uint64_t seed, uint64_t env_offset, uint64_t step, int n,
                        float* uniforms, void* stream) {
    CFX_REQUIRE(uniforms && n > 0, "cfx_philox_uniforms: bad argument");
    CFX_GUARD(device);
    return launch_uniforms(seed, env_offset, step, n, uniforms, (cudaStream_t)stream);
}

// ------------------------------------------------------------------ helpers
int cfx_device_count(int* count) {
    CFX_REQUIRE(count, "cfx_device_count: NULL");
    *count = 0;
    CFX_CUDA(cudaGetDeviceCount(count));
    return CFX_OK;
}

int cfx_device_name(int device, char* buf, size_t len, int* sm_count, int* cc_major, int* cc_minor) {
    cudaDeviceProp prop;
    CFX_CUDA(cudaGetDeviceProperties(&prop, device));
    if (buf && len) {
        strncpy(buf, prop.name, len - 1);
        buf[len - 1] = 0;
    }
    if (sm_count) *sm_count = prop.multiProcessorCount;
    if (cc_major) *cc_major = prop.major;
    if (cc_minor) *cc_minor = prop.minor;
    return CFX_OK;
}

int cfx_device_alloc(int device, void** ptr, size_t bytes) {
    CFX_REQUIRE(ptr, "cfx_device_alloc: NULL");
    CFX_GUARD(device);
    CFX_CUDA(cudaMalloc(ptr, bytes ? bytes : 1));
    return CFX_OK;
}

int cfx_device_free(int device, void* ptr) {
    CFX_GUARD(device);
    CFX_CUDA(cudaFree(ptr));
    return CFX_OK;
}

int cfx_host_alloc_pinned(void** ptr, size_t bytes) {
    CFX_REQUIRE(ptr, "cfx_host_alloc_pinned: NULL");
    CFX_CUDA(cudaMallocHost(ptr, bytes ? bytes : 1));
    return CFX_OK;
}

int cfx_host_free_pinned(void* ptr) {
    CFX_CUDA(cudaFreeHost(ptr));
    return CFX_OK;
}

int cfx_memcpy_h2d(int device, void* dst, const void* src, size_t bytes, void* stream) {
    CFX_GUARD(device);
    CFX_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, (cudaStream_t)stream));
    return CFX_OK;
}

int cfx_memcpy_d2h(int device, void* dst, const void* src, size_t bytes, void* stream) {
    CFX_GUARD(device);
    CFX_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    return CFX_OK;
}

int cfx_memset(int device, void* dst, int value, size_t bytes, void* stream) {
    CFX_GUARD(device);
    CFX_CUDA(cudaMemsetAsync(dst, value, bytes, (cudaStream_t)stream));
    return CFX_OK;
}

int cfx_stream_sync(int device, void* stream) {
    CFX_GUARD(device);
    CFX_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    return CFX_OK;
}

struct cfx_timer {
    int device;
    cudaEvent_t a, b;
};

int cfx_timer_create(int device, void** timer) {
    CFX_REQUIRE(timer, "cfx_timer_create: NULL");
    CFX_GUARD(device);
    cfx_timer* t = new (std::nothrow) cfx_timer();
    CFX_REQUIRE(t, "cfx_timer_create: out of host memory");
    t->device = device;
    CFX_CUDA(cudaEventCreate(&t->a));
    CFX_CUDA(cudaEventCreate(&t->b));
    *timer = t;
    return CFX_OK;
}

int cfx_timer_destroy(void* timer) {
    cfx_timer* t = (cfx_timer*)timer;
    if (!t) return CFX_OK;
    DeviceGuard g(t->device);
    cudaEventDestroy(t->a);
    cudaEventDestroy(t->b);
    delete t;
    return CFX_OK;
}

int cfx_timer_start(void* timer, void* stream) {
    cfx_timer* t = (cfx_timer*)timer;
    CFX_REQUIRE(t, "cfx_timer_start: NULL");
    CFX_GUARD(t->device);
    CFX_CUDA(cudaEventRecord(t->a, (cudaStream_t)stream));
    return CFX_OK;
}

int cfx_timer_stop(void* timer, void* stream) {
    cfx_timer* t = (cfx_timer*)timer;
    CFX_REQUIRE(t, "cfx_timer_stop: NULL");
    CFX_GUARD(t->device);
    CFX_CUDA(cudaEventRecord(t->b, (cudaStream_t)stream));
    return CFX_OK;
}

int cfx_timer_elapsed_ms(void* timer, float* ms) {
    cfx_timer* t = (cfx_timer*)timer;
    CFX_REQUIRE(t && ms, "cfx_timer_elapsed_ms: NULL");
    CFX_GUARD(t->device);
    CFX_CUDA(cudaEventSynchronize(t->b));
    CFX_CUDA(cudaEventElapsedTime(ms, t->a, t->b));
    return CFX_OK;
}

}  // extern "C"
