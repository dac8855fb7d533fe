"""Record writes where their tiles and copies end: views over the edges of the map, every alignment of the map
planes and of the records, blocks with and without skipped envs, batches that end inside a block."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PLANE = 9 * 48 * 48


def _view(cfx, st, shift, pad):
    """An EnvView whose maps start `shift` bytes into blocks of 3 * PLANE + shift + pad bytes."""
    n = st["player_level"].shape[1]
    view, keep = cfx.env_view_from_state(st)
    stride = 3 * PLANE + shift + pad
    blocks = np.zeros((n, stride), np.uint8)
    for k, m in enumerate(cfx.ENV_VIEW_MAPS):
        blocks[:, shift + k * PLANE:shift + (k + 1) * PLANE] = st[m].reshape(n, PLANE)
    d = cfx.DeviceBuffer.from_host(blocks)
    view.state_base, view.state_stride = d.ptr, stride
    view.map_offset, view.item_map_offset, view.light_map_offset = (shift + k * PLANE for k in range(3))
    return view, keep + [d]


@pytest.mark.parametrize("shift,pad,rec_shift", [(0, 0, 0), (16, 0, 4), (4, 8, 0), (4, 0, 12), (1, 0, 0), (2, 3, 4)])
@pytest.mark.parametrize("n", [1, 31, 33, 100])
def test_record_rows_at_edges(cfx, gpu, oracle, n, shift, pad, rec_shift):
    st = oracle.synthetic_env_state(n, seed=n)
    rng = np.random.default_rng(n + shift)
    edge = np.array([-40, -10, -9, -5, -4, -1, 0, 1, 4, 5, 24, 42, 43, 44, 46, 47, 48, 52, 53, 60, 100])
    st["player_position"][:] = rng.choice(edge, (2, n))
    st["mob_position"][:] = (st["player_position"][None] + rng.integers(-6, 7, (135, 2, n))).reshape(270, n)
    want = oracle.record_from_state(st)
    view, keep = _view(cfx, st, shift, pad)
    rec = cfx.DeviceBuffer((n * 996 + 16,), np.uint8)

    def at(offset):
        class Ref:
            ptr = rec.ptr + offset
        return Ref
    for skip in (None, (rng.random(n) < 0.1).astype(np.uint8)):
        rec.fill(0xCD)
        cfx.record_obs(view, at(rec_shift), skip=None if skip is None else cfx.DeviceBuffer.from_host(skip))
        cfx.check(cfx.lib().cfx_stream_sync(0, None))
        raw = rec.download()
        got = raw[rec_shift:rec_shift + n * 996].reshape(n, 996)
        done = np.ones(n, bool) if skip is None else skip == 0
        assert np.array_equal(got[done], want[done]) and (got[~done] == 0xCD).all()
        assert (raw[:rec_shift] == 0xCD).all() and (raw[rec_shift + n * 996:] == 0xCD).all()
        if skip is not None:   # the rest by the list
            lst = np.full((n, 3), -7, np.int32)
            which = np.nonzero(skip)[0]
            lst[:which.size, 0] = which
            cfx.record_obs_list(view, at(rec_shift), cfx.DeviceBuffer.from_host(lst), 12,
                                cfx.DeviceBuffer.from_host(np.array([which.size], np.int32)))
            cfx.check(cfx.lib().cfx_stream_sync(0, None))
            assert np.array_equal(rec.download()[rec_shift:rec_shift + n * 996].reshape(n, 996), want)
    del keep


@pytest.mark.parametrize("shift", [0, 4, 1])
def test_record_rows_at_every_column(cfx, gpu, oracle, shift):
    """Every column of the player, on, beside and off the map, so every alignment of a view's rows to words and to 16 bytes."""
    rows, cols = np.meshgrid([-5, 0, 3, 24, 44, 47, 52], np.arange(-7, 56), indexing="ij")
    n = rows.size
    st = oracle.synthetic_env_state(n, seed=5)
    st["player_position"][:] = np.stack([rows.ravel(), cols.ravel()])
    st["mob_position"][:] = (st["player_position"][None] + np.random.default_rng(shift).integers(-6, 7, (135, 2, n))).reshape(270, n)
    view, keep = _view(cfx, st, shift, 0)
    rec = cfx.DeviceBuffer((n, 996), np.uint8)
    cfx.record_obs(view, rec)
    cfx.check(cfx.lib().cfx_stream_sync(0, None))
    assert np.array_equal(rec.download(), oracle.record_from_state(st))
    del keep


CLASSIC_FIELDS = (("player_r", "i2", 1), ("player_c", "i2", 1), ("player_dir", "i1", 1), ("health", "i1", 1), ("food", "i1", 1),
                  ("drink", "i1", 1), ("energy", "i1", 1), ("is_sleeping", "u1", 1), ("inv", "i1", 12),
                  ("zombie_r", "i2", 3), ("zombie_c", "i2", 3), ("zombie_mask", "u1", 3), ("cow_r", "i2", 3),
                  ("cow_c", "i2", 3), ("cow_mask", "u1", 3), ("skel_r", "i2", 2), ("skel_c", "i2", 2),
                  ("skel_mask", "u1", 2), ("arrow_r", "i2", 3), ("arrow_c", "i2", 3), ("arrow_mask", "u1", 3),
                  ("light_level", "f4", 1))


class ClassicView(C.Structure):
    _fields_ = [("num_envs", C.c_int32), ("map_packed", C.c_void_p), ("map_stride", C.c_uint64)] + \
               [(name, C.c_void_p) for name, _, _ in CLASSIC_FIELDS]


def _classic_records(f, maps):
    """craftax_classic.cu:1574-1604, :1061-1126, env by env."""
    n = maps.shape[0]
    rec = np.zeros((n, 148), np.uint8)
    for e in range(n):
        pr, pc = int(f["player_r"][0, e]), int(f["player_c"][0, e])
        for r in range(7):
            for c in range(9):
                mr, mc = pr - 3 + r, pc - 4 + c
                b = 1
                if 0 <= mr < 64 and 0 <= mc < 64:
                    b = maps[e, mr * 32 + mc // 2] >> (4 * (mc & 1)) & 15
                rec[e, r * 9 + c] = b
        for kind, (name, slots) in enumerate((("zombie", 3), ("cow", 3), ("skel", 2), ("arrow", 3))):
            for i in range(slots):
                dr, dc = int(f[name + "_r"][i, e]) - pr + 3, int(f[name + "_c"][i, e]) - pc + 4
                if f[name + "_mask"][i, e] and 0 <= dr < 7 and 0 <= dc < 9:
                    rec[e, 63 + dr * 9 + dc] |= 1 << kind
        rec[e, 126:138] = f["inv"][:, e].view(np.uint8)
        for k, name in enumerate(("health", "food", "drink", "energy", "player_dir")):
            rec[e, 138 + k] = f[name][:, e].view(np.uint8)[0]
        rec[e, 143] = f["is_sleeping"][0, e] != 0
        rec[e, 144:] = f["light_level"][:, e:e + 1].copy().view(np.uint8)
    return rec


@pytest.mark.parametrize("n,stride,rec_shift", [(1, 2048, 0), (127, 2052, 4), (128, 2049, 0), (259, 2048, 12),
                                                (64, 2064, 0), (65, 2048, 0)])
def test_classic_record_rows_at_edges(cfx, gpu, n, stride, rec_shift):
    rng = np.random.default_rng(n)
    maps = rng.integers(0, 256, (n, stride)).astype(np.uint8)
    edge = np.array([-9, -4, -3, -1, 0, 1, 2, 3, 4, 5, 30, 31, 32, 33, 58, 59, 60, 61, 62, 63, 64, 67, 80])
    f = {}
    for name, dt, count in CLASSIC_FIELDS:
        if name in ("player_r", "player_c"):
            a = rng.choice(edge, (count, n))
        elif name[-2:] in ("_r", "_c"):
            a = f["player" + name[-2:]] + rng.integers(-5, 6, (count, n))
        elif name == "light_level":
            a = rng.random((count, n))
        else:
            a = rng.integers(0, 2, (count, n)) if name.endswith("mask") or name == "is_sleeping" else rng.integers(-3, 10, (count, n))
        f[name] = np.ascontiguousarray(a.astype(dt))
    d_map = cfx.DeviceBuffer.from_host(maps)
    view, keep = ClassicView(), []
    view.num_envs, view.map_packed, view.map_stride = n, d_map.ptr, stride
    for name, _, _ in CLASSIC_FIELDS:
        keep.append(cfx.DeviceBuffer.from_host(f[name]))
        setattr(view, name, keep[-1].ptr)
    rec = cfx.DeviceBuffer((n * 148 + 16,), np.uint8)
    rec.fill(0xCD)
    cfx.check(cfx.lib().cfx_classic_record_obs(0, C.byref(view), rec.ptr + rec_shift, n, None))
    cfx.check(cfx.lib().cfx_stream_sync(0, None))
    raw = rec.download()
    assert np.array_equal(raw[rec_shift:rec_shift + n * 148].reshape(n, 148), _classic_records(f, maps))
    assert (raw[:rec_shift] == 0xCD).all() and (raw[rec_shift + n * 148:] == 0xCD).all()
