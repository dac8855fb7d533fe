"""Performance cases of the library: what a rollout or training program has it do, through the
Python binding (`craftax.cu_b200/cfx`), over the range of batch sizes, shapes and operand types
that the repository's configurations, sweep and tests use.

Kinds of case:
  act       one policy step on records that are on the GPU (cfx_policy_forward), full game
  train     the same, with the BPTT record of the recurrent state that a trainer asks for
  host      the same from host buffers, copies in both directions included (cfx_policy_forward_host)
  classic   one policy step of the classic game
  record    the record write of a rollout step: all rows but those of the envs that are being
            reset, then the listed rows (cfx_record_obs with skip flags, cfx_record_obs_list)
  classic_record   the record write of the classic game

Run with the repository's root as the working folder.  `n` is the number of envs (a multiple of
32 for the policy, as its entry points require).
"""
import functools
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("craftax.cu_b200"))
import cfx  # noqa: E402

ACTIONS = {"full": 43, "classic": 17}
FEATURES = {"full": cfx.OBS, "classic": cfx.CLASSIC_OBS}
RECORD = {"full": cfx.REC, "classic": cfx.CLASSIC_REC}
END_SHARE = 1.0 / 265.0   # share of the envs whose episode ended in the step before


def listed():
    return [
        # the smallest rollouts of the reference's own table (1,024 envs), where latency counts
        dict(name="act-1k", kind="act", n=1024, hidden=256, layers=2, precision="f16"),
        # its training batch: half of the chip is idle when a tile has an SM of its own
        dict(name="act-8k", kind="act", n=8192, hidden=256, layers=2, precision="f16"),
        # the middle of the range at depth 3: a few tiles for every SM, and a last wave
        dict(name="act-64k-x3", kind="act", n=65536, hidden=256, layers=3, precision="f16"),
        # the headline batch
        dict(name="act-256k", kind="act", n=262144, hidden=256, layers=2, precision="f16"),
        # the narrow policy with bf16 operands, a batch that is not whole tiles
        dict(name="act-128k-h128-bf16", kind="act", n=131104, hidden=128, layers=2, precision="bf16"),
        # a step whose state inputs are kept for the backward pass, ragged batch
        dict(name="train-16k", kind="train", n=16416, hidden=256, layers=2, precision="f16", r_state="bf16"),
        # the accuracy mode: what a run is verified against
        dict(name="fp32-4k", kind="act", n=4096, hidden=256, layers=2, precision="fp32"),
        # the wide policy of the sweep, which only the fp32 mode runs
        dict(name="fp32-8k-h512x3", kind="act", n=8192, hidden=512, layers=3, precision="fp32"),
        # an evaluation or inference loop whose envs live on the host
        dict(name="host-64k", kind="host", n=65536, hidden=256, layers=2, precision="f16"),
        # the classic game at its headline batch
        dict(name="classic-1m-x3", kind="classic", n=1048576, hidden=256, layers=3, precision="f16"),
        # the record half of a rollout step, full game
        dict(name="record-64k", kind="record", n=65536),
        # and of the classic game
        dict(name="classic-record-256k", kind="classic_record", n=262144),
    ]


def _log_size(rng, lo, hi, step):
    """A multiple of `step` in [lo, hi], spread over the logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random() / step)) * step))


def draw(rng):
    kind = rng.choice(["act", "act", "act", "train", "fp32", "host", "classic", "record", "classic_record"])
    if kind == "record":
        return dict(kind=kind, n=_log_size(rng, 32, 65536, 1))
    if kind == "classic_record":
        return dict(kind=kind, n=_log_size(rng, 32, 262144, 1))
    if kind == "fp32":
        hidden = rng.choice([64, 128, 256, 512])
        return dict(kind="act", n=_log_size(rng, 32, 8192, 32), hidden=hidden, layers=rng.randint(1, 3),
                    precision="fp32")
    precision = rng.choice(["f16", "f16", "bf16"])
    layers = rng.randint(1, 3)
    if kind == "classic":
        return dict(kind=kind, n=_log_size(rng, 32, 1048576, 32), hidden=256, layers=layers, precision=precision)
    case = dict(kind=kind, n=_log_size(rng, 32, 65536 if kind == "host" else 262144, 32),
                hidden=rng.choice([256, 256, 128]), layers=layers, precision=precision)
    if kind == "train":
        case["r_state"] = rng.choice(["fp32", "bf16"])
    return case


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=None)
def rollout_stream():
    """The stream a rollout queues its steps on: each step starts where the one before it ended."""
    return torch.cuda.Stream()


class Ref:
    """What the binding takes for a device buffer: anything with a `ptr`."""

    def __init__(self, tensor):
        self.tensor, self.ptr = tensor, tensor.data_ptr()


class DeviceView:
    """The policy's recurrent state as an array on the GPU; keeps the policy alive."""

    def __init__(self, pol):
        self.pol = pol
        self.__cuda_array_interface__ = {"shape": (pol.L, pol.n, pol.H), "typestr": "<f4", "version": 2,
                                         "data": (cfx.lib().cfx_policy_state(pol.h), False)}


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _ints(g, lo, hi, shape, dtype=torch.int32):
    return torch.randint(lo, hi, shape, generator=g, device="cuda", dtype=dtype)


def _chance(g, p, shape):
    return torch.rand(shape, generator=g, device="cuda") < p


def _weights(game, H, L, seed):
    """N(0, 1/fan_in) weights, small biases, in the order of the parameter arena."""
    A, F = ACTIONS[game], FEATURES[game]
    rng = np.random.default_rng(seed)
    active = 85.0 if game == "classic" else float(F)   # features of a record that are not zero
    parts = [(F * H, active ** -0.5), (H, 0.05), (L * 3 * H * H, H ** -0.5), (A * H, H ** -0.5), (A, 0.05),
             (H, H ** -0.5), (1, 0.05)]
    return np.concatenate([rng.standard_normal(count, dtype=np.float32) * np.float32(s) for count, s in parts])


def _full_records(g, n):
    """Full-game records: 99 cells of {block, item + 1, lit, five mob classes}, dark cells zero,
    a mob on a few cells, then 51 floats of which most are multiples of a tenth."""
    rec = torch.empty((n, cfx.REC), dtype=torch.uint8, device="cuda")
    cells = torch.zeros((n, 99, 8), dtype=torch.uint8, device="cuda")
    cells[:, :, 0] = _ints(g, 0, 37, (n, 99), torch.uint8)
    cells[:, :, 1] = 1 + _ints(g, 1, 6, (n, 99), torch.uint8) * _chance(g, 0.02, (n, 99))
    cells[:, :, 2] = 1
    cells[:, :, 3:] = _ints(g, 1, 9, (n, 99, 5), torch.uint8) * _chance(g, 0.01, (n, 99, 5))
    cells *= _chance(g, 0.9, (n, 99, 1))
    rec[:, :cfx.MAP] = cells.view(n, cfx.MAP)
    tail = _ints(g, 0, 11, (n, cfx.TAIL)).float() * 0.1
    rec[:, cfx.MAP:] = tail.view(torch.uint8)
    return rec


def _classic_records(g, n):
    """Classic records: 63 block ids, 63 mob bit masks, 16 counts, direction, sleeping, light."""
    rec = torch.empty((n, cfx.CLASSIC_REC), dtype=torch.uint8, device="cuda")
    rec[:, :63] = _ints(g, 0, 17, (n, 63), torch.uint8)
    rec[:, 63:126] = (1 << _ints(g, 0, 4, (n, 63), torch.uint8)) * _chance(g, 0.04, (n, 63))
    rec[:, 126:142] = _ints(g, 0, 10, (n, 16), torch.uint8)
    rec[:, 142] = _ints(g, 1, 5, (n,), torch.uint8)
    rec[:, 143] = _chance(g, 0.05, (n,))
    rec[:, 144:] = torch.rand((n, 1), generator=g, device="cuda").view(torch.uint8)
    return rec


def _policy(case, seed, g):
    game = "classic" if case["kind"] == "classic" else "full"
    n, H, L = case["n"], case["hidden"], case["layers"]
    pol = cfx.Policy(n, H, L, ACTIONS[game], case["precision"], game=game)
    pol.set_weights(_weights(game, H, L, seed))
    state = torch.as_tensor(DeviceView(pol), device="cuda")
    state.normal_(generator=g)
    ended = _chance(g, END_SHARE, (n,)).float()
    records = _classic_records(g, n) if game == "classic" else _full_records(g, n)
    return pol, game, state, ended, records


def _prepare_act(case, seed, g):
    pol, game, state, ended, records = _policy(case, seed, g)
    n, A = case["n"], ACTIONS[game]

    def empty(shape, dtype):
        return torch.empty(shape, dtype=dtype, device="cuda")
    out = {"actions": empty((n,), torch.int32), "env_actions": empty((n,), torch.float32),
           "logprobs": empty((n,), torch.float32), "values": empty((n,), torch.float32)}
    call = {"bump_step": True, "seed": seed, "stream": rollout_stream().cuda_stream}
    if case["kind"] == "train":
        bf16 = case["r_state"] == "bf16"
        out["r_state"] = empty((pol.L, n, pol.H), torch.bfloat16 if bf16 else torch.float32)
        call["r_state_bf16"] = bf16
    else:
        out["logits_av"] = empty((n, A + 1), torch.float32)
    call.update({k: Ref(v) for k, v in out.items()})
    # the env's action slots hold whole numbers as floats: compared bit by bit
    result = dict(out, env_actions=out["env_actions"].view(torch.int32), state=state)
    return {"pol": pol, "records": Ref(records), "ended": Ref(ended), "call": call, "result": result}


def _prepare_host(case, seed, g):
    pol, game, state, ended, records = _policy(case, seed, g)
    n, A = case["n"], ACTIONS[game]

    def pinned(shape, dtype):
        return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()
    out = {"actions": pinned((n,), torch.int32), "env_actions": pinned((n,), torch.float32),
           "logprobs": pinned((n,), torch.float32), "values": pinned((n,), torch.float32),
           "logits_av": pinned((n, A + 1), torch.float32)}
    result = dict(out, env_actions=out["env_actions"].view(np.int32), state=state)
    return {"pol": pol, "records": records.cpu().pin_memory().numpy(), "ended": ended.cpu().pin_memory().numpy(),
            "out": out, "seed": seed, "result": result}


def _prepare_record(case, g):
    """The env state behind a rollout's record write: most envs on the first level, mobs around
    the player, about four in a thousand envs being reset."""
    n = case["n"]
    keep, view = [], cfx.EnvView()
    maps = torch.empty((n, 3, cfx.ENV_MAP_BYTES), dtype=torch.uint8, device="cuda")
    maps[:, 0].random_(0, 37, generator=g)           # block ids
    maps[:, 1].random_(0, 256, generator=g)          # items: on few cells
    maps[:, 1].mul_(maps[:, 1] < 6)
    maps[:, 2].random_(0, 256, generator=g)          # light: about one cell in twenty is dark
    view.num_envs, view.state_base, view.state_stride = n, maps.data_ptr(), 3 * cfx.ENV_MAP_BYTES
    view.map_offset, view.item_map_offset, view.light_map_offset = (k * cfx.ENV_MAP_BYTES for k in range(3))
    keep.append(maps)
    fields = {name: _ints(g, 0, 10, (count, n)) for name, _, count in cfx.ENV_VIEW_FIELDS}
    fields["player_position"] = _ints(g, 0, 48, (2, n))
    deep = _ints(g, 1, 9, (1, n))
    fields["player_level"] = torch.where(_chance(g, 0.85, (1, n)), torch.zeros_like(deep), deep)
    fields["player_direction"] = _ints(g, 1, 5, (1, n))
    fields["player_health"] = _ints(g, 1, 10, (1, n)).float()
    fields["light_level"] = torch.rand((1, n), generator=g, device="cuda")
    fields["mob_mask"] = _chance(g, 0.4, (135, n))
    fields["mob_type_id"] = _ints(g, 0, 8, (135, n))
    around = fields["player_position"][None] + _ints(g, -10, 11, (135, 2, n))
    fields["mob_position"] = around.clamp_(0, 47).view(270, n)
    types = {"i4": torch.int32, "f4": torch.float32, "u1": torch.uint8}
    for name, dtype, count in cfx.ENV_VIEW_FIELDS:
        t = fields[name]
        t = t.to(torch.bool) if name in ("is_sleeping", "is_resting", "learned_spells") else t
        t = t.to(types[dtype]).contiguous()
        setattr(view, name, t.data_ptr())
        keep.append(t)
    reset = _chance(g, END_SHARE, (n,))
    which = torch.nonzero(reset).to(torch.int32)
    entries = torch.zeros((n, 3), dtype=torch.int32, device="cuda")   # 12-byte entries, env index first
    entries[:which.shape[0], :1] = which
    count = torch.tensor([which.shape[0]], dtype=torch.int32, device="cuda")
    records = torch.empty((n, cfx.REC), dtype=torch.uint8, device="cuda")
    return {"view": view, "keep": keep, "skip": Ref(reset.to(torch.uint8)), "entries": Ref(entries),
            "count": Ref(count), "records": Ref(records)}


class ClassicView(cfx.C.Structure):
    """cfx_classic_env_view of include/cfx.h."""
    FIELDS = (("player_r", "i2", 1), ("player_c", "i2", 1), ("player_dir", "i1", 1), ("health", "i1", 1),
              ("food", "i1", 1), ("drink", "i1", 1), ("energy", "i1", 1), ("is_sleeping", "u1", 1), ("inv", "i1", 12),
              ("zombie_r", "i2", 3), ("zombie_c", "i2", 3), ("zombie_mask", "u1", 3),
              ("cow_r", "i2", 3), ("cow_c", "i2", 3), ("cow_mask", "u1", 3),
              ("skel_r", "i2", 2), ("skel_c", "i2", 2), ("skel_mask", "u1", 2),
              ("arrow_r", "i2", 3), ("arrow_c", "i2", 3), ("arrow_mask", "u1", 3), ("light_level", "f4", 1))
    _fields_ = [("num_envs", cfx.C.c_int32), ("map_packed", cfx.C.c_void_p), ("map_stride", cfx.C.c_uint64)] + \
               [(name, cfx.C.c_void_p) for name, _, _ in FIELDS]


CLASSIC_MAP_BYTES = 64 * 32


def _prepare_classic_record(case, g):
    n = case["n"]
    keep, view = [], ClassicView()
    blocks = _ints(g, 0, 256, (n, CLASSIC_MAP_BYTES), torch.uint8)   # two block ids a byte
    view.num_envs, view.map_packed, view.map_stride = n, blocks.data_ptr(), CLASSIC_MAP_BYTES
    keep.append(blocks)
    row, col = _ints(g, 0, 64, (1, n)), _ints(g, 0, 64, (1, n))
    types = {"i2": torch.int16, "i1": torch.int8, "u1": torch.uint8, "f4": torch.float32}
    for name, dtype, count in ClassicView.FIELDS:
        if name in ("player_r", "player_c"):
            t = row if name == "player_r" else col
        elif name.endswith("_r") or name.endswith("_c"):
            t = ((row if name.endswith("_r") else col) + _ints(g, -10, 11, (count, n))).clamp_(0, 63)
        elif name.endswith("_mask"):
            t = _chance(g, 0.4, (count, n))
        elif name == "is_sleeping":
            t = _chance(g, 0.05, (count, n))
        elif name == "light_level":
            t = torch.rand((count, n), generator=g, device="cuda")
        elif name == "player_dir":
            t = _ints(g, 1, 5, (count, n))
        else:
            t = _ints(g, 0, 10, (count, n))
        t = t.to(types[dtype]).contiguous()
        setattr(view, name, t.data_ptr())
        keep.append(t)
    records = torch.empty((n, cfx.CLASSIC_REC), dtype=torch.uint8, device="cuda")
    return {"view": view, "keep": keep, "records": Ref(records)}


# ------------------------------------------------------------------ the interface
def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "record":
        s = _prepare_record(case, g)
    elif kind == "classic_record":
        s = _prepare_classic_record(case, g)
    elif kind == "host":
        s = _prepare_host(case, seed, g)
    else:
        s = _prepare_act(case, seed, g)
    torch.cuda.synchronize()   # what was prepared is there before another stream reads it
    return dict(s, kind=kind)


def run(s):
    kind = s["kind"]
    if kind == "record":
        stream = rollout_stream().cuda_stream
        cfx.record_obs(s["view"], s["records"], skip=s["skip"], stream=stream)
        cfx.record_obs_list(s["view"], s["records"], s["entries"], 12, s["count"], stream=stream)
        return s["records"].tensor
    if kind == "classic_record":
        cfx.check(cfx.lib().cfx_classic_record_obs(0, cfx.C.byref(s["view"]), s["records"].ptr, s["view"].num_envs,
                                                   rollout_stream().cuda_stream))
        return s["records"].tensor
    if kind == "host":
        s["pol"].forward_host(s["records"], s["ended"], seed=s["seed"], bump_step=True, out=s["out"])
    else:
        s["pol"].forward_device(s["records"], s["ended"], **s["call"])
    return s["result"]


def work(case):
    n, kind = case["n"], case["kind"]
    if kind == "record":
        # 99 cells in three byte maps, 48 words of scalars, 14 mob slots of 13 bytes, the flag;
        # the record written once
        return {"bytes": n * (3 * 99 + 4 * 48 + 14 * 13 + 1 + cfx.REC), "flops": 0}
    if kind == "classic_record":
        # 63 cells of a nibble, 26 bytes of scalars, 11 mob slots of 5 bytes
        return {"bytes": n * (32 + 26 + 11 * 5 + cfx.CLASSIC_REC), "flops": 0}
    game = "classic" if kind == "classic" else "full"
    H, L, A = case["hidden"], case["layers"], ACTIONS[game]
    # the classic encoder is a sum of about 98 columns of its matrix (63 blocks, a few mobs, 22 scalars)
    inputs = 98 if game == "classic" else FEATURES[game]
    flops = n * (2 * inputs * H + 6 * L * H * H + 2 * (A + 1) * H)
    weights = FEATURES[game] * H + 3 * L * H * H + (A + 1) * H
    per_env = RECORD[game] + 8 * L * H + 4 + 16   # record, state in and out, terminal flag, four outputs
    if kind == "train":
        per_env += L * H * (2 if case["r_state"] == "bf16" else 4)
    else:
        per_env += 4 * (A + 1)
    return {"bytes": n * per_env + weights * (4 if case["precision"] == "fp32" else 2), "flops": flops}


def tolerance(case):
    if case["kind"] in ("record", "classic_record"):
        return "exact"
    # operands of 11 and 8 significant bits with fp32 accumulation; fp32 sums.  An action differs
    # where a probability's rounding moves a boundary of the distribution across its uniform.
    return {"f16": {"rel": 2e-3, "differ": 2e-3}, "bf16": {"rel": 1.5e-2, "differ": 1e-2},
            "fp32": {"rel": 1e-5, "differ": 1e-4}}[case["precision"]]
