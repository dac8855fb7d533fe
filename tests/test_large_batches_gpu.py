"""Calls that take another way for many envs, on both sides of where it changes: the record write of a long list."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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
