"""LayerNorm and head sums of rows of 64, 128 and 256 channels against 64 bits: one row, rows that leave a step of the lane groups and a warp's
steps incomplete, and one more than the resident grid takes in a pass.  A value is some 2^3 roundings of 2^-24 in the normalisation and a sum
of c products, in a tree over lanes of at most 2^5 terms each: 2^-18 of sum |x||w| covers c = 256."""
import pytest
import torch

from tt_boltz_b200 import _lib
from tt_boltz_b200.ops import ptr, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads", [4, 8, 16])
@pytest.mark.parametrize("c, passes, rest", [(64, 0, 1), (64, 0, 13), (64, 1, 3), (128, 0, 7), (128, 1, 1), (256, 0, 3), (256, 1, 1)])
def test_against_64_bits(c, passes, rest, heads):
    # a pass of the resident grid: two blocks of eight warps a multiprocessor, each with eight, four and four rows at a time
    rows = passes * torch.cuda.get_device_properties(0).multi_processor_count * 2 * 8 * (8 if c == 64 else 4) + rest
    torch.manual_seed(rows + heads)
    dev = "cuda:0"
    x = torch.randn(rows, c, device=dev) * 3 + torch.randn(rows, 1, device=dev)
    gamma, beta, w = torch.rand(c, device=dev) + 0.5, torch.randn(c, device=dev), torch.randn(heads, c, device=dev) * 0.1
    out = torch.full((heads, rows + 3), 7.0, device=dev)
    _lib.call("b200pf_ln_heads", ptr(x), ptr(gamma), ptr(beta), ptr(w), ptr(out), rows + 3, rows, c, heads, stream())
    torch.cuda.synchronize()
    xn = torch.nn.functional.layer_norm(x.double(), (c,), gamma.double(), beta.double(), 1e-5)
    unit = (x.double().abs() + x.double().mean(1, keepdim=True).abs()) * torch.rsqrt(x.double().var(1, unbiased=False, keepdim=True) + 1e-5)
    size = w.double().abs() @ (unit * gamma.double() + beta.double().abs()).T
    assert ((out[:, :rows].double() - w.double() @ xn.T).abs() <= 2.0 ** -18 * size).all()
    assert (out[:, rows:] == 7).all()
