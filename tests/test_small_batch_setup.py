"""Set-up of the small-batch kernel against a fake CUDA runtime: what the compiler gave the kernel decides whether it is used,
never whether a policy can be made."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OBJECT = os.path.join(ROOT, "craftax.cu_b200", "build", "cfx_fused_split.o")

FAKE = r"""
#include "cfx.h"
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
static int g_regs;
namespace cfx {
void set_error(const char*, ...) {}
int cuda_fail(cudaError_t, const char*, const char*, int) { return CFX_ERR_CUDA; }
namespace fused { int split_prepare(int precision, int game, int H, int S, int sm_count, int* max_clusters); }
}
extern "C" {
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaErrorUnknown; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { return cudaErrorUnknown; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { *a = {}; a->numRegs = g_regs; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) { *n = 33; return cudaSuccess; }
}
int main(int, char** argv) {
    g_regs = atoi(argv[1]);
    int clusters = -1;
    const int rc = cfx::fused::split_prepare(CFX_PREC_F16, CFX_GAME_FULL, 256, atoi(argv[2]), 148, &clusters);
    printf("%d %d\n", rc, clusters);
}
"""


@pytest.fixture(scope="module")
def program(cfx, tmp_path_factory):
    if not os.path.exists(OBJECT):
        import build
        build.build(force=True)
    d = tmp_path_factory.mktemp("split")
    src, exe = d / "fake.cpp", d / "fake"
    src.write_text(FAKE)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "include"), "-I", os.path.join(cuda, "include"), str(src), OBJECT,
                    "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("registers,ctas,clusters", [(96, 4, 33), (102, 4, 33), (95, 4, 0), (88, 4, 0), (88, 2, 33)])
def test_too_few_registers_leave_the_kernel_out(program, registers, ctas, clusters):
    """(Two CTAs a tile keep the registers they were launched with.)"""
    out = subprocess.run([program, str(registers), str(ctas)], capture_output=True, text=True, check=True).stdout.split()
    assert [int(x) for x in out] == [0, clusters]
