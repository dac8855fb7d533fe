"""The check build: every wrapper of an asynchronous copy verifies its operands there."""
import os
import re

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
