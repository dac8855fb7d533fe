"""The check build: every wrapper of an asynchronous copy verifies its operands there."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "craftax.cu_b200", "csrc")


def test_every_copy_wrapper_checks_its_operands():
    src = open(os.path.join(CSRC, "cfx_umma.cuh")).read()
    functions = re.split(r"\n(?=(?:template <[^\n]*\n)?__device__ __forceinline__ )", src)
    copies = [f for f in functions if re.search(r'"cp\.async\.bulk\.(?!commit|wait)', f)]
    assert len(copies) >= 7
    missing = [f.split("(")[0].split()[-1] for f in copies if "CFX_CHK(" not in f]
    assert not missing, missing


def test_the_policy_kernels_issue_copies_through_the_wrappers_only():
    for name in ("cfx_fused.cu", "cfx_fused_split.cu", "cfx_fused_common.cuh"):
        assert "cp.async.bulk" not in open(os.path.join(CSRC, name)).read(), name


def test_a_barrier_of_any_cta_of_a_cluster_passes_the_check(tmp_path):
    """In a cluster a CTA's own shared addresses carry its rank above the offset.  A check that refuses them skips the set-up of
    the barriers of every CTA but the first, and their users then run on barriers that were never set up."""
    src = tmp_path / "barrier.cu"
    src.write_text("""#define CFX_CHECK
#include "cfx_umma.cuh"
using cfx::umma::own_barrier;
constexpr bool in_every_cta(uint32_t offset) {
    for (uint32_t rank = 0; rank < 16; rank++)
        if (!own_barrier(rank << 24 | offset)) return false;
    return true;
}
static_assert(in_every_cta(1024) && in_every_cta(0x38800) && in_every_cta(233472 - 8), "own barriers");
static_assert(!own_barrier(1028) && !own_barrier(233472) && !own_barrier(1u << 24 | 233472), "not barriers");
""")
    subprocess.run(["nvcc", "-std=c++17", "-arch=sm_100a", "-I", CSRC, "-c", str(src), "-o", str(tmp_path / "barrier.o")], check=True)
    header = open(os.path.join(CSRC, "cfx_umma.cuh")).read()
    checks = re.findall(r'CFX_CHK(?:_BOOL)?\((.*?), "mbar_', header)
    assert len(checks) >= 5 and all(c == "own_barrier(bar)" for c in checks), checks
