"""The persistent kernel's data slots, which hold a tile's records and then the state boxes of its layers, over several tiles a
CTA: layers that leave slots without a box (hidden 128, one layer) or use some of them more often than others (three), the classic
game's records beside the boxes, a last tile of 32 and of 96 rows.  Bit for bit what the small-batch form, which has no such
slots, computes for slices of the batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _two_steps(cfx, H, L, prec, game, rec, params, state, prev_t, first):
    n, A = len(rec), 17 if game == "classic" else 43
    pol = cfx.Policy(n, H, L, A, prec, game=game)
    pol.set_weights(params)
    pol.set_state(state)
    pol.step = 5
    out = {"actions": cfx.DeviceBuffer((n,), np.int32), "logprobs": cfx.DeviceBuffer((n,), np.float32),
           "values": cfx.DeviceBuffer((n,), np.float32), "logits_av": cfx.DeviceBuffer((n, A + 1), np.float32)}
    d_rec, d_pt = cfx.DeviceBuffer.from_host(rec), cfx.DeviceBuffer.from_host(prev_t)
    for _ in range(2):   # the second step reads what the first one wrote
        pol.forward_device(d_rec, d_pt, seed=3, env_offset=first, bump_step=True, **out)
    pol.check()
    got = dict({k: b.download() for k, b in out.items()}, state=pol.get_state())
    pol.close()
    return got


@pytest.mark.parametrize("n,H,L,prec,game", [
    (56864, 128, 1, "f16", "full"), (38016, 128, 3, "bf16", "full"), (75872, 128, 2, "f16", "full"),
    (56928, 256, 1, "bf16", "full"), (37984, 256, 4, "f16", "full"), (56928, 256, 1, "f16", "classic"), (38016, 256, 4, "bf16", "classic")])
def test_several_tiles_a_cta_equal_small_batches(cfx, gpu, n, H, L, prec, game):
    from cfx import synth
    classic = game == "classic"
    m = 4096
    rec = (synth.classic_synthetic_records if classic else synth.synthetic_records)(m, seed=n)[np.arange(n) * 7 % m]
    params = synth.classic_init_weights(H, L, 17, seed=1) if classic else synth.init_weights(H, L, 43, seed=1)
    rng = np.random.default_rng(n)
    state = rng.standard_normal((L, n, H), dtype=np.float32)
    prev_t = (rng.random(n) < 0.2).astype(np.float32)
    got = _two_steps(cfx, H, L, prec, game, rec, params, state, prev_t, 0)
    for first in (0, 18944, 37888 - 512, n - 1024):   # tiles of the first, second and third round, and the last ones
        s = slice(first, first + 1024)
        if s.stop > n:
            continue
        want = _two_steps(cfx, H, L, prec, game, rec[s], params, np.ascontiguousarray(state[:, s]), prev_t[s], first)
        for k in want:
            assert np.array_equal(got[k][:, s] if k == "state" else got[k][s], want[k]), (k, first)
