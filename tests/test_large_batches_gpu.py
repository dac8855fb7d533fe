"""Calls that take another kernel for many envs, on both sides of where it changes: the stand-alone sampler, and the
record write of a long list of envs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65535, 65536, 65537, 131071, 131200])
@pytest.mark.parametrize("A,pad", [(2, 0), (17, 0), (32, 1), (33, 0), (43, 1), (63, 0)])
def test_sampler_rule(cfx, gpu, n, A, pad):
    """The same arithmetic in the same order in both forms: a batch is sampled as its halves are."""
    rng = np.random.default_rng(n + A)
    logits = rng.normal(0, 2, (n, A + pad)).astype(np.float32)
    logits[::97, 0] = -np.inf
    logits[5::101, A - 1] = np.inf     # no action has a probability: the last one
    logits[7::103, A // 2] = np.nan
    u = rng.random(n, dtype=np.float32)
    u[::11], u[1::11] = 0.0, np.float32(1.0)

    def sample(lo, hi):
        d_l, d_u = cfx.DeviceBuffer.from_host(logits[lo:hi]), cfx.DeviceBuffer.from_host(u[lo:hi])
        a, lp = cfx.DeviceBuffer((hi - lo + 1,), np.int32), cfx.DeviceBuffer((hi - lo + 1,), np.float32)
        a.fill(0xCD), lp.fill(0xCD)
        cfx.check(cfx.lib().cfx_sample_actions(0, d_l.ptr, A + pad, A, d_u.ptr, hi - lo, a.ptr, lp.ptr, None))
        cfx.check(cfx.lib().cfx_stream_sync(0, None))
        a, lp = a.download(), lp.download()
        assert a.view(np.uint32)[-1] == 0xCDCDCDCD and lp.view(np.uint32)[-1] == 0xCDCDCDCD
        return a[:-1], lp[:-1]
    parts = [sample(lo, min(lo + 50000, n)) for lo in range(0, n, 50000)]
    a, lp = sample(0, n)
    assert np.array_equal(a, np.concatenate([p[0] for p in parts]))
    assert np.array_equal(lp, np.concatenate([p[1] for p in parts]), equal_nan=True)


@pytest.mark.parametrize("entries,shift", [(2 * 2368, 0), (2 * 2368 + 1, 0), (6001, 4), (2 * 2368 + 33, 1)])
def test_record_list_rule(cfx, gpu, oracle, entries, shift):
    """Entry for entry what the reference writes, also entries outside the batch (left out) and envs named twice."""
    n, plane = 9472, 9 * 48 * 48    # so many that the grid of the list pass is full
    m = 256                          # the state of 256 envs over and over
    st = oracle.synthetic_env_state(m, seed=3)
    rng = np.random.default_rng(entries)
    st["player_position"][:] = rng.integers(-3, 51, (2, m))
    want = oracle.record_from_state(st)
    times = n // m
    view, keep = cfx.env_view_from_state({k: (np.tile(v, (1, times)) if v.ndim == 2 and v.shape[1] == m else np.tile(v, (times,) + (1,) * (v.ndim - 1)))
                                          for k, v in st.items()})
    stride = 3 * plane + 8
    blocks = np.zeros((m, stride), np.uint8)
    for k, name in enumerate(cfx.ENV_VIEW_MAPS):
        blocks[:, shift + k * plane:shift + (k + 1) * plane] = st[name].reshape(m, plane)
    d = cfx.DeviceBuffer.from_host(np.tile(blocks, (times, 1)))
    view.state_base, view.state_stride = d.ptr, stride
    view.map_offset, view.item_map_offset, view.light_map_offset = (shift + k * plane for k in range(3))
    which = rng.permutation(n)[:entries].astype(np.int32)
    which[[0, 40, entries - 1]] = -1, n, which[1]
    lst = np.full((entries, 3), -7, np.int32)
    lst[:, 0] = which
    rec = cfx.DeviceBuffer((n, 996), np.uint8)
    rec.fill(0xCD)
    cfx.record_obs_list(view, rec, cfx.DeviceBuffer.from_host(lst), 12, cfx.DeviceBuffer.from_host(np.array([entries], np.int32)))
    cfx.check(cfx.lib().cfx_stream_sync(0, None))
    got, named = rec.download(), np.zeros(n, bool)
    named[which[(which >= 0) & (which < n)]] = True
    assert np.array_equal(got[named], np.tile(want, (times, 1))[named])
    assert (got[~named] == 0xCD).all()
    del keep
