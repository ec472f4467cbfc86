"""The pair transition's two kernels: one tile of 128 rows per CTA, and CTA pairs that share the weights over several tiles.  Rows are
independent, so what a row comes to may not depend on the kernel or the tile it went through: at one tile more and one less than there are
multiprocessors, with an odd tile for the pairs, rows short of a tile, and many tiles per pair, each row equals, to the bit, what it comes
to in launches of at most 64 tiles, and those agree with torch in 64 bits (bf16 operands at three places: 2^-9 each, 1e-2 of the update's
norm together)."""
import pytest
import torch
import torch.nn.functional as F

from tt_boltz_b200 import B200PairformerModule, _lib, ops, synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def packed():
    mod = B200PairformerModule(384, 128, 1, v2=True)
    sd = synthetic.make_weights(1, seed=3, std=0.05, affine_jitter=0.2)
    mod.load_state_dict(sd, strict=True)
    return mod, {k.split("transition_z.")[1]: v.cuda().double() for k, v in sd.items() if "transition_z." in k}


def _rows(name):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return {"one row": 1, "short tile": 77, "all but one": (sms - 1) * 128 + 1, "all": sms * 128, "one more": sms * 128 + 1, "odd": (sms + 3) * 128 - 5,
            "many": 5 * sms * 128 + 200}[name]


@pytest.mark.parametrize("name", ["one row", "short tile", "all but one", "all", "one more", "odd", "many"])
def test_rows_are_independent_of_their_kernel(packed, name):
    mod, sd = packed
    w, n = mod.layers[0]._pack(torch.device("cuda:0"))["transition_z"], _rows(name)
    z = torch.randn(1, n, 128, generator=torch.Generator().manual_seed(n)).cuda()
    got = z.clone()
    ops.transition_z_bf16(got, w)
    want = z.clone()
    for r in range(0, n, 64 * 128):
        part = want[:, r:r + 64 * 128].contiguous()
        ops.transition_z_bf16(part, w)
        want[:, r:r + 64 * 128] = part
    assert _lib.device_status() == 0
    assert torch.equal(got, want)
    head = z[0, :4000].double()
    x = F.layer_norm(head, (128,), sd["norm.weight"], sd["norm.bias"], 1e-5)
    upd = (F.silu(x @ sd["fc1.weight"].t()) * (x @ sd["fc2.weight"].t())) @ sd["fc3.weight"].t()
    assert float(((want[0, :4000].double() - head) - upd).norm() / upd.norm()) < 1e-2
