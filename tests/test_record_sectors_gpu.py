"""The bf16 record of the state, which the cells write a 32-byte sector a thread where it starts on one: the same bits where it starts 16 bytes on,
nothing written beside it, in every form of the forward."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
A, GUARD = 43, 64   # 16-bit values in front of the record and behind it


class At:
    def __init__(self, ptr):
        self.ptr = ptr


# small batches with 32, 64 and 128 rows a tile, four CTAs and two; persistent, one tile a CTA and several, an odd number of them
@pytest.mark.parametrize("n,H,L,prec,pair", [
    (96, 256, 2, "f16", "1"), (1088, 256, 1, "f16", "1"), (2112, 256, 3, "bf16", "1"), (2144, 256, 2, "f16", "1"), (4256, 256, 4, "bf16", "1"),
    (4768, 256, 2, "f16", "1"), (9472, 256, 1, "bf16", "1"), (9504, 256, 2, "f16", "1"), (19104, 256, 3, "bf16", "1"), (9504, 256, 2, "f16", "0"),
    (2400, 128, 2, "f16", "1"), (9504, 128, 1, "f16", "1"), (19104, 128, 4, "bf16", "1"), (9504, 128, 3, "bf16", "0")])
def test_sectors_hold_the_record(cfx, gpu, monkeypatch, n, H, L, prec, pair):
    from cfx import synth
    monkeypatch.setenv("CFX_FUSED_PAIR", pair)
    rng = np.random.default_rng(n)
    rec = cfx.DeviceBuffer.from_host(synth.synthetic_records(n, seed=1))
    state = rng.standard_normal((L, n, H), dtype=np.float32)
    state[:, ::7, ::5] *= np.float32(1e-3)
    ended = (rng.random(n) < 0.2).astype(np.float32)
    ended[:3] = 1
    d_ended = cfx.DeviceBuffer.from_host(ended)
    want = state.copy()
    want[:, ended != 0] = 0
    u = want.view(np.uint32).astype(np.uint64)
    want = ((u + 0x7FFF + ((u >> 16) & 1)) >> 16).astype(np.uint16)
    pol = cfx.Policy(n, H, L, A, prec)
    pol.set_weights(synth.init_weights(H, L, A, seed=1))
    outs = []
    for offset in (0, 8):
        buf = cfx.DeviceBuffer.from_host(np.full(want.size + 2 * GUARD, 0x5A5A, np.uint16))
        out = {"actions": cfx.DeviceBuffer((n,), np.int32), "logits_av": cfx.DeviceBuffer((n, A + 1), np.float32)}
        pol.set_state(state)
        first = GUARD + offset
        assert (buf.ptr + 2 * GUARD) % 32 == 0
        pol.forward_device(rec, d_ended, seed=3, r_state_bf16=True, r_state=At(buf.ptr + 2 * first), **out)
        pol.check()
        got = buf.download()
        assert np.array_equal(got[first:first + want.size].reshape(want.shape), want)
        assert (got[:first] == 0x5A5A).all() and (got[first + want.size:] == 0x5A5A).all()
        outs.append((out["logits_av"].download(), pol.get_state()))
    for a, b in zip(*outs):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    pol.close()


@pytest.mark.parametrize("n,L,prec", [(2400, 3, "bf16"), (4224, 4, "bf16"), (3232, 1, "f16")])
def test_records_off_a_sector_of_four_ctas_a_tile(cfx, gpu, monkeypatch, n, L, prec):
    """Where the record starts off a sector four CTAs have a tile of 128 rows, on one two have 64: the same bits."""
    test_sectors_hold_the_record(cfx, gpu, monkeypatch, n, 256, L, prec, "1")
