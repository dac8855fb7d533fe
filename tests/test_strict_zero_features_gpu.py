"""fp32 encoder: features that are zero in all envs of a block are left out, which changes no bit of a result and nothing where a weight is
not finite."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
A, L, MAP = 43, 1, 792


def _forward(cfx, params, rec, n, H):
    pol = cfx.Policy(n, H, L, A, "fp32")
    pol.set_weights(params)
    d = pol.forward_host(rec, None, np.full(n, 0.5, np.float32))
    out = dict(logits=d["logits_av"].copy(), state=pol.get_state()[0])
    pol.close()
    return out


# a size for every form of the kernel (see test_strict_tiles_gpu.py): one sum a lane, 4 units, 4 and more envs a lane, warps along units or envs
@pytest.mark.parametrize("n,H", [(32, 256), (160, 256), (416, 256), (1632, 256), (4128, 256), (2528, 512), (1056, 96), (5408, 192)])
# features left: none, the first or last one, and with the tail of 51 a stage's end (16 or 32 rows) less one, met and passed by one
@pytest.mark.parametrize("kept", [[], [0], [MAP - 1], range(12), range(13), range(14), range(5, MAP, 7), range(MAP)],
                         ids=["none", "first", "last", "63", "64", "65", "seventh", "all"])
def test_left_out_features_change_no_bit(cfx, gpu, oracle, n, H, kept):
    rng = np.random.default_rng(n + H)
    params = oracle.init_weights(H, L, A, seed=5, scheme="uniform")
    kept = np.array(kept, int)
    rec = oracle.synthetic_records(n, seed=4)
    mask = np.zeros(MAP, bool)
    mask[kept] = True
    rec[:, :MAP] *= mask
    # every feature is there in one env only, which another one of the block may have
    own = rng.integers(0, n, MAP)
    rec[:, :MAP] *= (np.arange(n)[:, None] % 16 == own[None] % 16)
    got = _forward(cfx, params, rec, n, H)
    lav = oracle.forward(params, rec, None, np.zeros((L, n, H), np.float32), H, L, A)
    assert np.abs(got["logits"] - lav).max() < 3e-5 * max(1.0, np.abs(lav).max())
    # the same envs in blocks that leave nothing out: each fourth one has every feature
    full = rec.copy()
    full[::4, :MAP] = 1
    want = _forward(cfx, params, full, n, H)
    same = np.arange(n) % 4 != 0
    for k in got:
        assert np.array_equal(got[k][same], want[k][same]), k


@pytest.mark.parametrize("n,H", [(32, 256), (416, 256), (4128, 256)])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_weights_that_are_not_finite_reach_every_env(cfx, gpu, oracle, n, H, value):
    """0 times such a weight is not a number: the unit is lost in all envs, also where the feature is zero in all of them; and the next
    weights are looked at anew."""
    params = oracle.init_weights(H, L, A, seed=5, scheme="uniform")
    rec = oracle.synthetic_records(n, seed=4)
    rec[:, 700] = 0
    bad = params.copy()
    bad[700 * H + H - 1] = value
    pol = cfx.Policy(n, H, L, A, "fp32")
    want = None
    for p in (params, bad, params):
        pol.set_weights(p)
        pol.reset_state()
        lav = pol.forward_host(rec, None, np.full(n, 0.5, np.float32))["logits_av"].copy()
        if p is bad:
            assert np.isnan(lav).all()
        elif want is None:
            want = lav
        else:
            assert np.array_equal(lav, want) and np.isfinite(lav).all()
    pol.close()


@pytest.mark.parametrize("n", [32, 416, 1024])
def test_each_static_forward_looks_at_its_own_weights(cfx, gpu, oracle, n):
    """Forwards of the allocation-free entry point one behind the other on a stream, with weights that are finite and that are not in turn: what
    the kernel in front of the encoder finds in them is what the encoder goes by."""
    H = 256
    params = oracle.init_weights(H, L, A, seed=5, scheme="uniform")
    rec = oracle.synthetic_records(n, seed=4)
    rec[:, 700] = 0
    bad = params.copy()
    bad[700 * H + H - 1] = np.inf
    weights = [cfx.DeviceBuffer.from_host(p) for p in (params, bad)]
    d_rec, d_state = cfx.DeviceBuffer.from_host(rec), cfx.DeviceBuffer((L, n, H), np.float32)
    d_u, d_act = cfx.DeviceBuffer.from_host(np.full(n, 0.5, np.float32)), cfx.DeviceBuffer((n,), np.int32)
    ended = cfx.DeviceBuffer.from_host(np.ones(n, np.float32))   # every forward starts from a state of zeros
    outs = [cfx.DeviceBuffer((n, A + 1), np.float32) for _ in range(40)]
    for i, out in enumerate(outs):
        io = cfx.ForwardIO(d_rec.ptr, ended.ptr, d_u.ptr, None, d_act.ptr, None, None, out.ptr, None, 0, 0, 0, 0)
        cfx.check(cfx.lib().cfx_strict_forward_static(0, weights[i % 2].ptr, H, L, A, n, d_state.ptr, C.byref(io), None, None))
    cfx.check(cfx.lib().cfx_stream_sync(0, None))
    want = outs[0].download()
    assert np.isfinite(want).all()
    for i, out in enumerate(outs):
        lav = out.download()
        assert np.isnan(lav).all() if i % 2 else np.array_equal(lav, want), i


@pytest.mark.parametrize("n,H", [(32, 256), (160, 256), (416, 256), (1632, 256), (2592, 256), (4128, 256), (2528, 512), (1056, 96), (4768, 64), (5408, 192)])
def test_records_without_zeros_give_the_bits_of_a_list(cfx, gpu, oracle, n, H):
    """Where nothing is left out the features are taken by words of the map: the same bits as where one is left out, whose weights are zero."""
    params = oracle.init_weights(H, L, A, seed=5, scheme="uniform")
    params[700 * H:701 * H] = 0
    rec = oracle.synthetic_records(n, seed=4)
    rec[:, :MAP] = np.maximum(rec[:, :MAP], 1)
    got = _forward(cfx, params, rec, n, H)
    lav = oracle.forward(params, rec, None, np.zeros((L, n, H), np.float32), H, L, A)
    assert np.abs(got["logits"] - lav).max() < 3e-5 * max(1.0, np.abs(lav).max())
    rec[:, 700] = 0
    want = _forward(cfx, params, rec, n, H)
    for k in got:
        assert np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)), k
