// Shared definitions of the B200 policy-forward library: constants of the
// record / arena layout, the handle, error plumbing.
#pragma once
#include <cuda_runtime.h>
#include <atomic>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include "../../include/cfx.h"

namespace cfx {

constexpr int kObs = CFX_OBS_FEATURES;   // 843 features
constexpr int kMap = CFX_OBS_MAP;        // 792 one-byte map features
constexpr int kTail = CFX_OBS_TAIL;      // 51 raw fp32 tail features
constexpr int kRec = CFX_RECORD_BYTES;   // 996-byte record
constexpr int kMaxActions = 63;
constexpr int kMaxHidden = 512;
// classic game (reference craftax_classic.cu:38-59): 148-byte record, 1345 features
constexpr int kClassicRec = CFX_CLASSIC_RECORD_BYTES, kClassicObs = CFX_CLASSIC_OBS_FEATURES;
constexpr int kClassicCells = 63, kClassicBlocks = 17, kClassicInv = 12;

// Arena offsets in floats (reference order, craftax_full.cu:9094-9102).
struct ArenaLayout {
    size_t w_enc, b_enc, w_gru, w_a, b_a, w_v, b_v, count;
    __host__ __device__ static ArenaLayout make(int H, int L, int A, int obs = kObs) {
        ArenaLayout o;
        o.w_enc = 0;
        o.b_enc = (size_t)obs * H;
        o.w_gru = o.b_enc + H;
        o.w_a = o.w_gru + (size_t)L * 3 * H * H;
        o.b_a = o.w_a + (size_t)A * H;
        o.w_v = o.b_a + A;
        o.b_v = o.w_v + H;
        o.count = o.b_v + 1;
        return o;
    }
};

// Thread-local error string behind cfx_last_error().
void set_error(const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what, const char* file, int line);

#define CFX_CUDA(call)                                                        \
    do {                                                                      \
        cudaError_t _e = (call);                                              \
        if (_e != cudaSuccess) return ::cfx::cuda_fail(_e, #call, __FILE__, __LINE__); \
    } while (0)

#define CFX_REQUIRE(cond, ...)                 \
    do {                                       \
        if (!(cond)) {                         \
            ::cfx::set_error(__VA_ARGS__);     \
            return CFX_ERR_INVALID;            \
        }                                      \
    } while (0)

// Scoped cudaSetDevice.  Entry points use CFX_GUARD, which returns an error when the device
// cannot be selected instead of carrying on with whatever device is current.
struct DeviceGuard {
    int prev = -1;
    bool ok = true;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        if (prev == dev) prev = -1;   // nothing to put back
        else ok = (cudaSetDevice(dev) == cudaSuccess);
    }
    ~DeviceGuard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

#define CFX_GUARD(dev)                                                                   \
    ::cfx::DeviceGuard _cfx_guard(dev);                                                  \
    do {                                                                                 \
        if (!_cfx_guard.ok) {                                                            \
            cudaGetLastError();                                                          \
            ::cfx::set_error("%s: cannot select CUDA device %d", __func__, (int)(dev));  \
            return CFX_ERR_CUDA;                                                         \
        }                                                                                \
    } while (0)

// The current context's number, unique in the process, or 0 where it cannot be told (before the first use of a device).
unsigned long long current_context_id();

// Kernels launched with programmatic stream serialisation: the launch and the start-up of a kernel run
// under the kernel in front of it in the stream, and it waits here until the results of that kernel are in
// memory.  Nothing that another kernel may have written is read before, and nothing of it by read-only loads (a
// `const __restrict__` parameter makes them): those are for memory that nobody writes while the kernel lives, and it lives
// from its launch on.  Only kernels of few blocks
// let the next one start early (launch_next_kernel): the blocks of a larger one would fill the SMs that this
// kernel's last blocks leave free and pile up there (fp32 forward, 4,096 envs: 227 us against 178; classic record
// write, 20,000 envs: 9.1 us against 4.2).
#ifdef __CUDACC__
__device__ __forceinline__ void launch_next_kernel() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous_kernel() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... Args>
int launch_chained(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    CFX_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
    return CFX_OK;
}

// A kernel's dynamic shared memory limit and its preference for shared memory over L1, set once per context (they go with it: after
// cudaDeviceReset they are set again).  kMost is the most that the kernel is ever launched with, one value a kernel: host
// threads that come here at the same time with different shapes all set the same.
// (`static`: a process that has loaded two builds of the library sets them for the kernels of each)
template <auto kernel, int kMost>
static int allow_smem() {
    static std::atomic<unsigned long long> done[64];   // ids of contexts, an id's place is id % 64
    const unsigned long long id = current_context_id();
    if (id != 0 && done[id % 64].load(std::memory_order_relaxed) == id) return CFX_OK;
    CFX_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost));
    CFX_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    if (id != 0) done[id % 64].store(id, std::memory_order_relaxed);
    return CFX_OK;
}
#endif

}  // namespace cfx
