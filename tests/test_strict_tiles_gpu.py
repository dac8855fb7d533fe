"""Every tile shape of the fp32 kernels against the CPU oracle, at batch sizes that end inside
a tile, and the allocation-free variant on arrays that are only 4-byte aligned.

The cases: (n, hidden, layers) and the tiles that the library takes for them, as cfx_selftest_strict_tiles gives them: envs
a lane of the layers (0: one sum a gate), whether with 4 they have three stages; envs a lane of the encoder (0: one
sum) and its groups of four units.  (tests/test_strict_tiles.py: that they are so, and that none is missing.)"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
A = 43


def _inputs(oracle, n, H, L):
    rng = np.random.default_rng(n + H)
    return (oracle.synthetic_records(n, seed=4), oracle.init_weights(H, L, A, seed=5, scheme="uniform"),
            rng.normal(0, 1, (L, n, H)).astype(np.float32), (rng.random(n) < 0.3).astype(np.float32),
            rng.random(n, dtype=np.float32))


def _close(got, want):
    # both sides sum in the same order; they differ in expf and its neighbours (2 ulp each), which
    # the layers pass on: 3e-5 of the largest value, as for the other shapes of this mode
    assert np.abs(got - want).max() < 3e-5 * max(1.0, np.abs(want).max())


TILES = {
    (32, 32, 1): (1, 0, 0, 1),                                      # one unit tile
    (416, 256, 1): (4, 1, 4, 1), (1632, 256, 2): (6, 0, 4, 2),
    (2592, 256, 1): (9, 0, 5, 2), (4128, 256, 2): (7, 0, 7, 2),     # the last blocks of the encoder are not full
    (1056, 96, 2): (4, 0, 4, 1), (11040, 96, 1): (8, 0, 4, 1)}      # odd multiples of 32: the layers' warps along the envs
HEIGHTS = {
    (1248, 256, 1): (5, 0, 4, 2), (1568, 256, 1): (6, 0, 4, 2), (2048, 256, 2): (7, 0, 4, 2), (2272, 256, 1): (8, 0, 4, 2),
    (2528, 256, 1): (9, 0, 5, 2),
    (1248, 512, 1): (9, 0, 5, 2), (1504, 512, 1): (6, 0, 6, 2), (1760, 512, 1): (6, 0, 6, 2), (2272, 512, 1): (8, 0, 8, 2),
    (2528, 512, 1): (9, 0, 9, 2),
    # odd multiples of 64: the encoder's warps along the envs
    (3872, 192, 1): (4, 0, 5, 2), (5408, 192, 1): (4, 0, 7, 2),
    (4768, 64, 1): (4, 1, 4, 2), (11872, 64, 1): (4, 0, 6, 2), (5536, 192, 1): (8, 0, 8, 2), (6304, 192, 1): (4, 0, 9, 2)}
SMALLEST = {
    (32, 64, 4): (0, 0, 0, 1), (64, 512, 1): (0, 0, 0, 1), (128, 256, 2): (0, 0, 0, 1), (160, 192, 1): (0, 0, 0, 1),
    (96, 96, 2): (1, 0, 0, 1), (160, 256, 2): (1, 0, 1, 1), (352, 256, 1): (1, 0, 1, 1), (160, 512, 1): (1, 0, 1, 1)}


@pytest.mark.parametrize("n,H,L", TILES)
def test_strict_tiles_match_the_oracle(cfx, gpu, oracle, n, H, L):
    rec, params, state, prev_t, u = _inputs(oracle, n, H, L)
    pol = cfx.Policy(n, H, L, A, "fp32")
    pol.set_weights(params)
    pol.set_state(state)
    pol.step = 7
    d = pol.forward_host(rec, prev_t, u, want_r_state=True, bump_step=True)
    st = state.copy()
    lav, rs = oracle.forward(params, rec, prev_t, st, H, L, A, want_r_state=True)
    _close(d["logits_av"], lav)
    _close(pol.get_state(), st)
    assert np.array_equal(d["r_state"], rs)
    assert pol.step == 8     # raised by the sampler's last block
    a, lp = oracle.sample(d["logits_av"][:, :A], u)
    assert (d["actions"] != a).sum() <= 1    # a boundary of the distribution within rounding of its uniform
    same = d["actions"] == a
    assert np.abs(d["logprobs"][same] - lp[same]).max() < 1e-5
    pol.close()


def test_static_forward_takes_arrays_of_any_word_alignment(cfx, gpu, oracle):
    n, H, L = 96, 256, 2
    rec, params, state, prev_t, u = _inputs(oracle, n, H, L)

    def shifted(a):   # device copy that starts 4 bytes past an aligned address
        return cfx.DeviceBuffer.from_host(np.concatenate([np.zeros(1, np.float32), a.ravel()]))
    d_par, d_st = shifted(params), shifted(state)
    d_rec, d_pt, d_u = (cfx.DeviceBuffer.from_host(x) for x in (rec, prev_t, u))
    d_act, d_lav = cfx.DeviceBuffer((n,), np.int32), cfx.DeviceBuffer((n, A + 1), np.float32)
    io = cfx.ForwardIO(d_rec.ptr, d_pt.ptr, d_u.ptr, None, d_act.ptr, None, None, d_lav.ptr, None, 0, 0, 0, 0)
    cfx.check(cfx.lib().cfx_strict_forward_static(0, d_par.ptr + 4, H, L, A, n, d_st.ptr + 4, C.byref(io), None, None))
    cfx.check(cfx.lib().cfx_stream_sync(0, None))
    st = state.copy()
    lav = oracle.forward(params, rec, prev_t, st, H, L, A)
    _close(d_lav.download(), lav)
    _close(d_st.download()[1:].reshape(st.shape), st)


@pytest.mark.parametrize("n,H,L", HEIGHTS)
def test_strict_heights_match_the_oracle(cfx, gpu, oracle, n, H, L):
    """Heights that are no multiple of four envs a lane, and batches that end inside a block."""
    test_strict_tiles_match_the_oracle(cfx, gpu, oracle, n, H, L)


@pytest.mark.parametrize("n,H,L", SMALLEST)
def test_smallest_strict_batches_match_the_oracle(cfx, gpu, oracle, n, H, L):
    """One sum a lane, then two envs x two units in the layers, up to the last sizes that take them, and hidden sizes for which only
    the encoder does."""
    test_strict_tiles_match_the_oracle(cfx, gpu, oracle, n, H, L)


@pytest.mark.parametrize("n,H", [(32, 32), (32, 256), (416, 256), (1248, 256)])
def test_strict_saturated_gates(cfx, gpu, oracle, n, H):
    """Pre-activations up to some thousands: 1 + exp(-z) overflows, where the quotients are 0."""
    rec, params, state, prev_t, u = _inputs(oracle, n, H, 1)
    gates = slice(844 * H, 844 * H + 3 * H * H)
    params[gates] *= 200.0
    pol = cfx.Policy(n, H, 1, A, "fp32")
    pol.set_weights(params)
    pol.set_state(state)
    d = pol.forward_host(rec, prev_t, u)
    st = state.copy()
    lav = oracle.forward(params, rec, prev_t, st, H, 1, A)
    assert np.isfinite(lav).all() and np.abs(st).max() > 200
    _close(d["logits_av"], lav)
    _close(pol.get_state(), st)
    pol.close()


@pytest.mark.parametrize("H", [256, 96])   # (96: the layers' warps along the envs)
def test_batches_of_any_size_give_the_same_bits(cfx, gpu, oracle, H):
    """An env's results do not depend on which tiles its batch takes."""
    rec, params, state, prev_t, u = _inputs(oracle, 4128, H, 2)

    def run(n):
        pol = cfx.Policy(n, H, 2, A, "fp32")
        pol.set_weights(params)
        pol.set_state(np.ascontiguousarray(state[:, :n]))
        d = dict(pol.forward_host(rec[:n], prev_t[:n], u[:n], want_r_state=True), state=pol.get_state())
        pol.close()
        return {k: v[:, :32] if k in ("state", "r_state") else v[:32] for k, v in d.items()}
    want = run(4128)
    for n in (32, 160, 416, 1248, 1568, 2592):
        got = run(n)
        for k in want:
            assert np.array_equal(got[k], want[k]), (n, k)
