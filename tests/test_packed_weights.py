"""What a module keeps of its weights between calls: copies of a module pack their own."""
import copy

import pytest
import torch

from tt_boltz_b200 import B200PairUpdateBlock
from tt_boltz_b200.pairformer import B200PairformerNoSeqLayer

CPU = torch.device("cpu")


def _modules():
    return [B200PairformerNoSeqLayer(64, precision="fp32"), B200PairUpdateBlock(64, 128)]


def _fill(module, seed=0):
    g = torch.Generator().manual_seed(seed)
    with torch.no_grad():
        for p in module.parameters():
            p.copy_(torch.randn(p.shape, generator=g))
    return module


@pytest.mark.parametrize("i", [0, 1])
def test_a_used_module_can_be_copied(i):
    module = _fill(_modules()[i])
    pack = module._pack(CPU)
    twin = copy.deepcopy(module)
    assert module._packed is pack and twin._packed is None
    for (name, a), (_, b) in zip(module.named_parameters(), twin.named_parameters()):
        assert torch.equal(a, b) and a.data_ptr() != b.data_ptr(), name


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["bf16", "fp32"])
def test_a_copy_of_a_used_module_gives_its_results(precision):
    from tt_boltz_b200 import B200PairformerModule, synthetic
    module = B200PairformerModule(384, 128, 2, v2=True, precision=precision)
    module.load_state_dict(synthetic.make_weights(2, seed=3, std=0.05, affine_jitter=0.2), strict=True)
    s, z = (t.cuda() for t in synthetic.make_inputs(33, seed=1))
    want = module(s, z)
    twin = copy.deepcopy(module)
    del module
    got = twin(s, z)
    assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])
