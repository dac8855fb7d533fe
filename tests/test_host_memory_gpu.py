"""cfx_policy_forward_host on host arrays that are page-locked in part: the kernels may use an array in place only where
one piece of page-locked memory holds all of it."""
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
H, L, A = 256, 2, 43
PAGE = mmap.PAGESIZE


@pytest.mark.parametrize("n", [32, 256])
@pytest.mark.parametrize("pieces", ["front", "all", "two", "none"])
def test_partly_registered_logits(cfx, gpu, oracle, n, pieces):
    import torch
    rt = torch.cuda.cudart()
    torch.cuda.init()
    rec = oracle.synthetic_records(n, seed=3)
    pol = cfx.Policy(n, H, L, A, "f16")
    pol.set_weights(oracle.init_weights(H, L, A, seed=2))
    want = pol.forward_host(rec, None, seed=5)
    size = n * (A + 1) * 4
    pages = -(-size // PAGE)
    mem = mmap.mmap(-1, (pages + 1) * PAGE)
    base = np.frombuffer(mem, np.uint8)
    first = base.ctypes.data
    spans = {"none": [], "all": [(0, pages)], "front": [(0, 1)], "two": [(0, 1), (1, pages - 1)]}[pieces]
    for a, k in spans:
        assert int(rt.cudaHostRegister(first + a * PAGE, k * PAGE, 0)) == 0
    try:
        logits = base[:size].view(np.float32).reshape(n, A + 1)
        logits[...] = -1.0
        pol.reset_state()
        got = pol.forward_host(rec, None, seed=5, out={"logits_av": logits})
        for k in want:
            assert np.array_equal(got[k], want[k]), k
    finally:
        for a, _ in spans:
            assert int(rt.cudaHostUnregister(first + a * PAGE)) == 0
        pol.close()
