"""A stack called under CUDA graph capture (after one plain call, which packs the weights) replays to the plain call's result bit for
bit: with the single track on its own stream, and with a single track of a width that the part-plane kernels are not built for, which
stays on the caller's stream."""
import pytest
import torch

from tt_boltz_b200 import B200PairformerModule, _lib, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c_s, heads", [(384, 16), (192, 8)])
@pytest.mark.parametrize("precision", ["bf16", "mxfp8", "fp32"])
def test_captured_call(c_s, heads, precision):
    module = B200PairformerModule(c_s, 128, 3, num_heads=heads, v2=True, precision=precision)
    module.load_state_dict(synthetic.make_weights(3, seed=3, std=0.05, affine_jitter=0.2, c_s=c_s, num_heads=heads), strict=True)
    s, z = (t.cuda() for t in synthetic.make_inputs(37, c_s=c_s, seed=2))
    want = module(s, z)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = module(s, z)
    for t in got:
        t.zero_()
    graph.replay()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert _lib.device_status() == 0
