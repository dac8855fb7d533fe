"""A switch of the operand type that is refused leaves the handle as it was: the next forward, on any stream, and a
graph captured before it use the operands that were there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
H, L, A = 256, 4, 43
TF32 = 3   # reserved: not built for any shape


@pytest.mark.parametrize("n,prec", [(64, "f16"), (64, "bf16"), (9504, "f16"), (64, "fp32")])
def test_refused_switch_leaves_the_operands(cfx, gpu, oracle, n, prec):
    import torch
    rec = cfx.DeviceBuffer.from_host(oracle.synthetic_records(n, seed=2))
    out = {"actions": cfx.DeviceBuffer((n,), np.int32), "logits_av": cfx.DeviceBuffer((n, A + 1), np.float32)}
    pol = cfx.Policy(n, H, L, A, prec)
    pol.set_weights(oracle.init_weights(H, L, A, seed=7))
    stream, results = torch.cuda.Stream(), []

    def forward():
        pol.forward_device(rec, None, seed=1, stream=stream.cuda_stream, **out)

    def collect():
        pol.check(stream.cuda_stream)
        results.append((out["actions"].download(), out["logits_av"].download(), pol.get_state()))
    pol.reset_state()
    forward()
    collect()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        forward()
    for _ in range(8):
        pol.reset_state()
        with pytest.raises(cfx.CfxError):
            pol.set_precision(TF32)
        forward()
        collect()
        pol.reset_state()
        with torch.cuda.stream(stream):
            graph.replay()
        collect()
    assert cfx.lib().cfx_policy_get_precision(pol.h) == cfx.PREC_NAMES[prec]
    for got in results[1:]:
        for a, b in zip(got, results[0]):
            assert np.array_equal(a, b)
    pol.close()
