"""A stack called under CUDA graph capture replays to the plain call's result bit for bit: with the single track on its own stream, and
with a single track of a width that the part-plane kernels are not built for, which stays on the caller's stream; as the module's first
call, which packs its weights; and after the weights and the workspace have changed."""
import pytest
import torch

from tt_boltz_b200 import B200PairformerModule, B200PairformerNoSeqModule, _lib, synthetic

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


def _template(c, precision):
    module = B200PairformerNoSeqModule(c, 2, precision=precision)
    module.load_state_dict(synthetic.make_weights(2, seed=3, std=0.05, affine_jitter=0.2, with_s=False, c_z=c), strict=True)
    return module.cuda(), synthetic.make_inputs(29, c_z=c, seed=4, with_s=False)[1].cuda()


@pytest.mark.parametrize("c, precision", [(64, "fp32"), (96, "fp32"), (128, "bf16")])
def test_first_call_is_captured(c, precision):
    module, z = _template(c, precision)
    want = module(z)
    module, z = _template(c, precision)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = module(z)
    assert torch.equal(module(z), want)         # the pack is there before the first replay
    graph.replay()
    assert torch.equal(got, want)


@pytest.mark.parametrize("c, precision", [(64, "fp32"), (128, "bf16")])
def test_a_replay_computes_with_what_was_captured(c, precision):
    module, z = _template(c, precision)
    want = module(z)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = module(z)
    with torch.no_grad():
        for p in module.parameters():
            if p.dim() == 2:                                # (LayerNorm gains and offsets are read where they are)
                p.mul_(0.5)
    module.reset_static_cache()
    other = module(z[:, :17, :17].contiguous())             # new packs, another token count's workspace
    taken = [torch.full((1 << 20,), float("nan"), device="cuda") for _ in range(64)]
    graph.replay()
    assert torch.equal(got, want) and torch.isfinite(other).all() and len(taken) == 64
