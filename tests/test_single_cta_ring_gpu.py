"""The weight ring of the persistent kernel with one CTA per tile: encoder blocks that are cut across stages (hidden 256) or
come two at a time (128), gate stages of two K blocks, several tiles a CTA, so that the ring's position at a tile's start
changes.  Bit for bit what the CTA pairs, which have another ring, compute."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _two_steps(cfx, H, L, prec, game, rec, params, state, prev_t):
    n, A = len(rec), 17 if game == "classic" else 43
    pol = cfx.Policy(n, H, L, A, prec, game=game)
    pol.set_weights(params)
    pol.set_state(state)
    out = {"actions": cfx.DeviceBuffer((n,), np.int32), "logprobs": cfx.DeviceBuffer((n,), np.float32),
           "values": cfx.DeviceBuffer((n,), np.float32), "logits_av": cfx.DeviceBuffer((n, A + 1), np.float32)}
    d_rec, d_pt = cfx.DeviceBuffer.from_host(rec), cfx.DeviceBuffer.from_host(prev_t)
    for _ in range(2):
        pol.forward_device(d_rec, d_pt, seed=3, bump_step=True, **out)
    pol.check()
    got = dict({k: b.download() for k, b in out.items()}, state=pol.get_state())
    pol.close()
    return got


@pytest.mark.parametrize("n,H,L,prec,game", [
    (9504, 256, 1, "f16", "full"), (38016, 256, 2, "bf16", "full"), (57056, 256, 3, "f16", "full"), (38016, 256, 4, "f16", "full"),
    (37984, 128, 1, "bf16", "full"), (57056, 128, 2, "f16", "full"), (38016, 128, 3, "f16", "full"),
    (57056, 256, 1, "f16", "classic"), (38016, 256, 2, "f16", "classic"), (38016, 256, 3, "bf16", "classic")])
def test_one_cta_per_tile_equals_pairs(cfx, gpu, monkeypatch, n, H, L, prec, game):
    from cfx import synth
    classic = game == "classic"
    m = 4096
    rec = (synth.classic_synthetic_records if classic else synth.synthetic_records)(m, seed=n)[np.arange(n) * 7 % m]
    params = synth.classic_init_weights(H, L, 17, seed=1) if classic else synth.init_weights(H, L, 43, seed=1)
    rng = np.random.default_rng(n)
    state = rng.standard_normal((L, n, H), dtype=np.float32)
    prev_t = (rng.random(n) < 0.2).astype(np.float32)
    want = _two_steps(cfx, H, L, prec, game, rec, params, state, prev_t)
    monkeypatch.setenv("CFX_FUSED_PAIR", "0")
    got = _two_steps(cfx, H, L, prec, game, rec, params, state, prev_t)
    for k in want:
        assert np.array_equal(got[k], want[k]), k
