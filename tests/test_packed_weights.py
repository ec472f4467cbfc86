"""What a module keeps of its weights between calls: copies of a module pack their own, and the fp32 tier sees weights that are changed
in place, as it does on the un-fused kernels, which read the parameters themselves."""
import copy

import pytest
import torch

from tt_boltz_b200 import B200PairUpdateBlock, _lib, weights
from tt_boltz_b200.pairformer import B200PairformerNoSeqLayer

CPU = torch.device("cpu")


def _modules():              # of a width whose pack a CPU can make: the part planes are packed on the GPU
    return [B200PairformerNoSeqLayer(96, pairwise_num_heads=3, precision="fp32"), B200PairUpdateBlock(96, 128)]


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
    pack["struct"] = weights.SplitPack(_lib.SplitTransitionWeights(c=96), [])        # as part planes have them
    twin = copy.deepcopy(module)
    assert module._packed is pack and twin._packed is None
    for (name, a), (_, b) in zip(module.named_parameters(), twin.named_parameters()):
        assert torch.equal(a, b) and a.data_ptr() != b.data_ptr(), name


@pytest.mark.parametrize("i", [0, 1])
def test_weights_changed_in_place_are_packed_anew(i):
    module = _fill(_modules()[i])
    pack = module._pack(CPU)
    assert module._pack(CPU) is pack
    with torch.no_grad():
        next(p for name, p in module.named_parameters() if name == "transition_z.fc3.weight").mul_(3.0)
    new = module._pack(CPU)
    assert new is not pack and module._pack(CPU) is new
    module.reset_static_cache()                          # for changes through .data
    assert module._pack(CPU) is not new


@pytest.mark.gpu
@pytest.mark.parametrize("c", [64, 96])                  # on part planes, on the un-fused kernels
def test_the_fp32_tier_computes_with_weights_changed_in_place(c):
    z = torch.randn(1, 21, 21, c, generator=torch.Generator().manual_seed(1)).cuda()
    module = _fill(B200PairUpdateBlock(c, 128)).cuda()
    module(z)
    with torch.no_grad():
        for p in module.parameters():
            p.mul_(0.5)
    other = B200PairUpdateBlock(c, 128)
    other.load_state_dict(module.state_dict())
    assert torch.equal(module(z), other.cuda()(z))


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


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["bf16", "fp32"])
def test_a_pack_is_there_for_calls_on_other_streams(precision):
    """The first call, which packs, stands behind 50 ms of other work on its stream; a second one on another stream gives its result."""
    from tt_boltz_b200 import B200PairformerNoSeqModule, synthetic
    module = B200PairformerNoSeqModule(128, 2, precision=precision)
    module.load_state_dict(synthetic.make_weights(2, seed=3, std=0.05, affine_jitter=0.2, with_s=False), strict=True)
    module = module.cuda()
    z = synthetic.make_inputs(33, seed=1, with_s=False)[1].cuda()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        torch.cuda._sleep(100_000_000)
        first = module(z)
    twin = copy.copy(module)                                 # shares the packed weights,
    twin._ws_cache = {}                                      # but not the workspace
    with torch.cuda.stream(b):
        second = twin(z)
    torch.cuda.synchronize()
    assert torch.equal(first, second)
