"""cfx_policy_forward_host at the sizes where it changes its way of moving the arrays: the kernel reading and writing
host memory in place or copies, page-locked and pageable arrays, slices; against the device-pointer call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
H, L, A = 256, 2, 43


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("n", [32, 256, 288, 2048, 2080, 8160, 8192, 65536])
def test_host_forward_equals_device_forward(cfx, gpu, oracle, n, pinned):
    rng = np.random.default_rng(n)
    rec = oracle.synthetic_records(min(n, 4096), seed=6)[rng.integers(0, min(n, 4096), n)]
    state = rng.standard_normal((L, n, H), dtype=np.float32)
    prev_t = (rng.random(n) < 0.2).astype(np.float32)
    u = rng.random(n, dtype=np.float32)
    pol = cfx.Policy(n, H, L, A, "f16")
    pol.set_weights(oracle.init_weights(H, L, A, seed=12))
    shapes = {"actions": ((n,), np.int32), "env_actions": ((n,), np.float32), "logprobs": ((n,), np.float32),
              "values": ((n,), np.float32), "logits_av": ((n, A + 1), np.float32)}
    dev = {k: cfx.DeviceBuffer(*v) for k, v in shapes.items()}
    keep = []

    def host(shape, dtype, src=None):
        b = cfx.PinnedBuffer(shape, dtype) if pinned else None
        keep.append(b)
        a = b.array if pinned else np.empty(shape, dtype)
        a[...] = 0xCD if src is None else src
        return a
    out = {k: host(*v) for k, v in shapes.items()}
    h_rec, h_pt, h_u = host((n, 996), np.uint8, rec), host((n,), np.float32, prev_t), host((n,), np.float32, u)
    for uniforms in (None, u):
        pol.set_state(state)
        pol.step = 4
        d_u = None if uniforms is None else cfx.DeviceBuffer.from_host(u)
        pol.forward_device(cfx.DeviceBuffer.from_host(rec), cfx.DeviceBuffer.from_host(prev_t), d_u, seed=3, bump_step=True, **dev)
        pol.check()
        want = dict({k: b.download() for k, b in dev.items()}, state=pol.get_state())
        pol.set_state(state)
        pol.step = 4
        pol.forward_host(h_rec, h_pt, None if uniforms is None else h_u, seed=3, bump_step=True, out=out)
        assert pol.step == 5
        for k in shapes:
            assert np.array_equal(out[k], want[k]), k
        assert np.array_equal(pol.get_state(), want["state"])
    pol.close()
