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


@pytest.mark.parametrize("n,pinned,launches", [(32, True, 2), (256, True, 2), (288, True, 1), (32, False, 1)])
def test_launches_of_a_small_call(cfx, gpu, oracle, n, pinned, launches):
    """Page-locked records of the smallest batches are fetched by a kernel of their own, which counts."""
    buf = cfx.PinnedBuffer((n, 996), np.uint8)
    buf.array[...] = oracle.synthetic_records(n, seed=3)
    pol = cfx.Policy(n, H, L, A, "f16")
    pol.forward_host(buf.array if pinned else np.array(buf.array), None, seed=5)
    assert pol.last_launches == launches
    pol.close()


@pytest.mark.parametrize("pageable", [None, "logits_av", "actions"])
def test_slices_with_pageable_outputs(cfx, gpu, oracle, pageable):
    """A sliced call reads its outputs back at the end where one of them is pageable: the same values."""
    n = 65536 + 4128
    rec = cfx.PinnedBuffer((n, 996), np.uint8)
    rec.array[...] = oracle.synthetic_records(2048, seed=6)[np.arange(n) % 2048]
    pol = cfx.Policy(n, H, L, A, "f16")
    pol.set_weights(oracle.init_weights(H, L, A, seed=12))
    want = pol.forward_host(np.array(rec.array), None, seed=3)
    shapes = {k: cfx.PinnedBuffer(v.shape, v.dtype) for k, v in want.items()}
    out = {k: np.full(b.shape, 7, b.dtype) if k == pageable else b.array for k, b in shapes.items()}
    pol.reset_state()
    pol.forward_host(rec.array, None, seed=3, out=out)
    for k in want:
        assert np.array_equal(out[k], want[k]), k
    pol.close()
