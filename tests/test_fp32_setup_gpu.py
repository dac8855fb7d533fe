"""The fp32 mode's one-time set-up (its kernels' shared-memory limits), in processes of their own: first calls with
different shapes from several host threads at once, and calls after the device was reset."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = """
import sys, threading
sys.path[:0] = [{root!r} + "/craftax.cu_b200", {root!r} + "/oracle"]
import numpy as np
import cfx
import oracle as O
rec = O.synthetic_records(32, seed=1)

def forward(H, A):
    pol = cfx.Policy(32, H, 1, A, "fp32")
    pol.set_weights(O.init_weights(H, 1, A, seed=1))
    out = [pol.forward_host(rec, None, seed=1)["logits_av"] for _ in range(2)][0]
    pol.close()
    return out
""".format(root=ROOT)


def _run(code):
    p = subprocess.run([sys.executable, "-c", PRELUDE + code], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, p.stdout[-2000:] + p.stderr[-2000:]


@pytest.mark.parametrize("shapes", [[(32, 43), (512, 63)], [(512, 63), (32, 2), (256, 43), (96, 17)]])
def test_first_calls_of_several_threads(cfx, gpu, shapes):
    for _ in range(3):
        _run(f"shapes = {shapes!r}\n" + """
gate, failed = threading.Barrier(len(shapes)), []

def work(H, A):
    pol = cfx.Policy(32, H, 1, A, "fp32")
    out = {"actions": np.empty(32, np.int32)}
    gate.wait()
    try:
        for _ in range(20):
            pol.forward_host(rec, None, seed=1, want_logits=False, out=out)
    except cfx.CfxError as e:
        failed.append(str(e))
    gate.wait()
threads = [threading.Thread(target=work, args=s) for s in shapes]
[t.start() for t in threads]
[t.join() for t in threads]
for s in shapes:
    forward(*s)
assert not failed, failed
""")


@pytest.mark.parametrize("H,A", [(32, 2), (512, 63)])
def test_calls_after_a_device_reset(cfx, gpu, H, A):
    """The limits go with the context: handles made after cudaDeviceReset set them again."""
    _run(f"H, A = {H}, {A}\n" + """
import ctypes, glob, os
import nvidia
runtime, = glob.glob(os.path.join(list(nvidia.__path__)[0], "cuda_runtime/lib/libcudart.so.1*"))
before = forward(H, A)
runtime = ctypes.CDLL(runtime)
assert runtime.cudaSetDevice(0) == 0 and runtime.cudaDeviceReset() == 0
assert np.array_equal(forward(H, A), before)
""")
