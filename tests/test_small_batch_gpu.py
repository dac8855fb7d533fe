"""The small-batch form of the fused forward (a tile shared by a cluster of two or four CTAs) against the form
with one CTA per tile, bit for bit, at the ends of its ranges: tiles of 32, 64 and 128 rows, clusters of
four and of two, rows beyond the batch, the last batch sizes before the forms change."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _forward(cfx, n, H, L, prec, game, rec, params, state, prev_t, r_state, launches=1):
    A = 17 if game == "classic" else 43
    pol = cfx.Policy(n, H, L, A, prec, game=game)
    pol.set_weights(params)
    out = {"actions": cfx.DeviceBuffer((n,), np.int32), "env_actions": cfx.DeviceBuffer((n,), np.float32),
           "logprobs": cfx.DeviceBuffer((n,), np.float32), "values": cfx.DeviceBuffer((n,), np.float32),
           "logits_av": cfx.DeviceBuffer((n, A + 1), np.float32)}
    if r_state:
        out["r_state"] = cfx.DeviceBuffer((L, n, H), np.uint16 if r_state == "bf16" else np.float32)
    d_rec, d_pt = cfx.DeviceBuffer.from_host(rec), cfx.DeviceBuffer.from_host(prev_t)
    results = []
    for _ in range(launches):
        pol.set_state(state)
        pol.step = 5
        for _ in range(2):   # the second step starts from the first one's state
            pol.forward_device(d_rec, d_pt, seed=3, bump_step=True, r_state_bf16=r_state == "bf16", **out)
        pol.check()
        assert pol.step == 7
        results.append(dict({k: b.download() for k, b in out.items()}, state=pol.get_state()))
    pol.close()
    return results


@pytest.mark.parametrize("n,H,L,prec,game,r_state", [
    # four CTAs a tile: 32 rows to 1,056 envs, 64 to 2,112, and to 4,224 128 where the state is recorded in fp32; else (also in bf16 on a 32-byte
    # boundary) two CTAs with 64 rows
    (32, 256, 1, "f16", "full", "fp32"), (96, 256, 4, "bf16", "full", "bf16"),
    (1184, 256, 2, "f16", "full", None), (1216, 256, 2, "f16", "full", "fp32"),
    (2336, 256, 3, "bf16", "full", "bf16"), (2400, 256, 2, "f16", "full", None),    # (two CTAs, 64 rows)
    # two CTAs a tile: 64 rows to 4,736, 128 to 9,472; then the persistent kernel
    (4704, 256, 4, "f16", "full", "fp32"), (4768, 256, 2, "f16", "full", "bf16"),
    (9472, 256, 3, "f16", "full", "fp32"), (9504, 256, 1, "f16", "full", None),
    # hidden 128, two CTAs: 32 rows to 2,368, 64 to 4,736, 128 to 9,472
    (64, 128, 2, "f16", "full", "bf16"), (2368, 128, 1, "bf16", "full", "fp32"), (2400, 128, 3, "bf16", "full", "fp32"), (9440, 128, 4, "f16", "full", None),
    # the classic game, as hidden 256: tiles of 32, 64, two CTAs with 64 and with 128
    (160, 256, 3, "f16", "classic", None), (1152, 256, 2, "bf16", "classic", "bf16"), (4736, 256, 2, "bf16", "classic", "fp32"),
    (9376, 256, 3, "f16", "classic", "bf16"),
    # without a record, both sides of the limits between four CTAs and two, and of 64 and 128 rows
    (2112, 256, 2, "f16", "full", None), (2144, 256, 3, "bf16", "full", None), (3232, 256, 1, "f16", "full", None), (4224, 256, 3, "f16", "full", None),
    (4256, 256, 2, "bf16", "full", None), (4768, 256, 2, "f16", "full", None), (3200, 256, 3, "f16", "classic", None),
    (2400, 256, 2, "f16", "full", "bf16")])   # the same batch with one that the cells write: two CTAs, 64 rows too
def test_small_batch_form_equals_one_cta_per_tile(cfx, gpu, monkeypatch, n, H, L, prec, game, r_state):
    from cfx import synth
    classic = game == "classic"
    rec = (synth.classic_synthetic_records if classic else synth.synthetic_records)(n, seed=n)
    params = synth.classic_init_weights(H, L, 17, seed=1) if classic else synth.init_weights(H, L, 43, seed=1)
    rng = np.random.default_rng(n)
    state = rng.standard_normal((L, n, H), dtype=np.float32)
    prev_t = (rng.random(n) < 0.2).astype(np.float32)
    # ten launches: a row that depends on which warp comes first shows up in one of them
    got = _forward(cfx, n, H, L, prec, game, rec, params, state, prev_t, r_state, launches=10)
    monkeypatch.setenv("CFX_FUSED_PAIR", "0")
    want, = _forward(cfx, n, H, L, prec, game, rec, params, state, prev_t, r_state)
    for g in got:
        for k in want:
            assert np.array_equal(g[k], want[k]), k


@pytest.mark.parametrize("n,L,prec,r_state", [
    (2112, 3, "f16", "bf16"),                                                         # four CTAs, 64 rows
    (2144, 3, "bf16", "bf16"), (4224, 1, "f16", "bf16"), (3232, 2, "f16", "fp32"),    # two CTAs, 64 rows
    (3200, 3, "f16", "fp32")])                                                        # four CTAs, 128 rows
def test_classic_game_with_a_record(cfx, gpu, monkeypatch, n, L, prec, r_state):
    test_small_batch_form_equals_one_cta_per_tile(cfx, gpu, monkeypatch, n, 256, L, prec, "classic", r_state)


@pytest.mark.parametrize("n,L,prec", [(2144, 4, "f16"), (2336, 3, "bf16"), (3136, 2, "f16"), (3232, 1, "bf16"), (4192, 4, "bf16"), (4224, 3, "f16")])
def test_four_ctas_a_tile_of_128_rows(cfx, gpu, monkeypatch, n, L, prec):
    """With an fp32 record, from the first batch of this form to the last; the last tile has 32, 64, 96 or all of its rows."""
    test_small_batch_form_equals_one_cta_per_tile(cfx, gpu, monkeypatch, n, 256, L, prec, "full", "fp32")
