"""Kernels that start under the kernel in front of them (launch_chained): `const __restrict__` parameters may be read by read-only loads, which
neither wait for that kernel nor see what it writes.  Only weights that no kernel of a forward writes are such parameters."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "craftax.cu_b200", "csrc")
# (the gate matrices Wt are written in front of a forward by k_transpose_gates: read by asynchronous copies alone, which come behind the wait)
WEIGHTS = {"W_enc", "b_enc", "Wt", "W_a", "b_a", "W_v", "b_v"}


def _kernels():
    found = {}
    for name in sorted(os.listdir(CSRC)):
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for kernel in set(re.findall(r"launch_chained\(\s*(k_\w+)", text)):
            definition = re.search(r"__global__[^;{]*?\b" + kernel + r"\s*\(([^;{]*?)\)\s*\{", text)
            found[kernel] = definition.group(1)
    return found


@pytest.mark.parametrize("kernel,parameters", _kernels().items(), ids=_kernels())
def test_only_weights_are_read_by_read_only_loads(kernel, parameters):
    names = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", parameters))
    assert names <= WEIGHTS, names - WEIGHTS


def test_the_forward_s_kernels_are_looked_at():
    assert {"k_encoder_fp32", "k_mingru_fp32", "k_mingru_small", "k_heads_fp32", "k_classic_encoder_fp32"} <= set(_kernels())
