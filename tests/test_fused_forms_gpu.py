"""The persistent kernel as CTA pairs, at sizes that the small-batch form does not take, and that form where its
clusters and tiles change: bit for bit what one CTA per tile computes, both operand types, both record types, filler
tiles and several tiles a CTA; and the record of the state inputs against what it is a copy of."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _steps(cfx, n, H, L, prec, game, rec, params, state, prev_t, r_state):
    A = 17 if game == "classic" else 43
    pol = cfx.Policy(n, H, L, A, prec, game=game)
    pol.set_weights(params)
    pol.set_state(state)
    pol.step = 5
    out = {"actions": cfx.DeviceBuffer((n,), np.int32), "env_actions": cfx.DeviceBuffer((n,), np.float32),
           "logprobs": cfx.DeviceBuffer((n,), np.float32), "values": cfx.DeviceBuffer((n,), np.float32),
           "logits_av": cfx.DeviceBuffer((n, A + 1), np.float32)}
    if r_state:
        out["r_state"] = cfx.DeviceBuffer((L, n, H), np.uint16 if r_state == "bf16" else np.float32)
    d_rec, d_pt = cfx.DeviceBuffer.from_host(rec), cfx.DeviceBuffer.from_host(prev_t)
    got = []
    for _ in range(2):
        pol.forward_device(d_rec, d_pt, seed=3, bump_step=True, r_state_bf16=r_state == "bf16", **out)
        pol.check()
        got.append(dict({k: b.download() for k, b in out.items()}, state=pol.get_state()))
    assert pol.step == 7
    pol.close()
    return got


def _bf16(x):
    """Round to nearest even, as the device's conversion."""
    b = np.ascontiguousarray(x, np.float32).view(np.uint32)
    return ((b + 0x7FFF + ((b >> 16) & 1)) >> 16).astype(np.uint16)


@pytest.mark.parametrize("n,H,L,prec,game,r_state", [
    (9504, 256, 2, "bf16", "full", "bf16"),       # 75 tiles, the last one a quarter full
    (16416, 256, 2, "f16", "full", "bf16"),       # 129 tiles: a filler tile in the last pair
    (19008, 256, 3, "bf16", "full", "fp32"),      # 149 tiles: one pair has two rounds
    (57600, 256, 1, "f16", "full", "fp32"),       # 450: three or four tiles a CTA
    (9600, 128, 4, "bf16", "full", "fp32"), (38016, 128, 2, "bf16", "full", None), (16416, 128, 2, "f16", "full", "bf16"),
    # where 33 clusters of four and 74 of two are resident: the last tiles of 32, 64 and 128 rows for four CTAs, the first
    # of 64 and 128 after them, the first, the last and a ragged one of 64 rows for two CTAs
    (1056, 256, 2, "f16", "full", "bf16"), (1088, 256, 1, "bf16", "full", None), (2112, 256, 3, "bf16", "full", "fp32"),
    (2144, 256, 2, "f16", "full", "bf16"), (4224, 256, 1, "f16", "full", "fp32"), (4256, 256, 2, "bf16", "full", "fp32"),
    (4512, 256, 3, "f16", "full", "bf16"), (4736, 256, 4, "f16", "full", None), (4576, 256, 3, "f16", "classic", "bf16"),
    (9504, 256, 3, "bf16", "classic", "bf16"), (38048, 256, 2, "f16", "classic", "fp32")])
def test_pairs_equal_one_cta_per_tile(cfx, gpu, monkeypatch, n, H, L, prec, game, r_state):
    from cfx import synth
    classic = game == "classic"
    m = 4096
    rec = (synth.classic_synthetic_records if classic else synth.synthetic_records)(m, seed=n)[np.arange(n) * 7 % m]
    params = synth.classic_init_weights(H, L, 17, seed=1) if classic else synth.init_weights(H, L, 43, seed=1)
    rng = np.random.default_rng(n)
    state = rng.standard_normal((L, n, H), dtype=np.float32)
    prev_t = (rng.random(n) < 0.2).astype(np.float32)
    got = _steps(cfx, n, H, L, prec, game, rec, params, state, prev_t, r_state)
    monkeypatch.setenv("CFX_FUSED_PAIR", "0")
    want = _steps(cfx, n, H, L, prec, game, rec, params, state, prev_t, r_state)
    for g, w in zip(got, want):
        for k in w:
            assert np.array_equal(g[k], w[k]), k
    if r_state:   # the state each step started from, zero where the episode had ended
        for g, start in zip(got, (state, got[0]["state"])):
            before = np.where(prev_t[None, :, None] != 0, np.float32(0), start)
            assert np.array_equal(g["r_state"], _bf16(before) if r_state == "bf16" else before)
