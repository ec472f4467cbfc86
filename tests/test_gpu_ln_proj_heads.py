"""LayerNorm and projection of pair rows to 16 heads against 64 bits: fewer rows than a warp takes, remainders of its 16 and of a CTA's 128,
and more rows than the grid takes in one pass (the rolling fetch and its end).  Each normalised value and weight is held to 2^-22 and a
product of their parts left out is as much again, the mean, the variance and a sum of 128 products add 2^-24 a step over some 2^4 steps of
a tree or a tensor instruction each: 2^-19 of sum |x||w| covers them all.  A row that holds a NaN is one in the result."""
import pytest
import torch

from tt_boltz_b200 import _lib
from tt_boltz_b200.ops import ptr, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("passes, rest", [(0, 1), (0, 15), (0, 17), (0, 127), (0, 129), (1, 5), (3, -1)])
def test_against_64_bits(passes, rest):
    rows = passes * torch.cuda.get_device_properties(0).multi_processor_count * 2 * 128 + rest      # two blocks of 128 rows a multiprocessor
    torch.manual_seed(rows)
    dev = "cuda:0"
    z = torch.randn(rows, 128, device=dev) * 3 + torch.randn(rows, 1, device=dev)
    gamma, beta, w = torch.rand(128, device=dev) + 0.5, torch.randn(128, device=dev), torch.randn(16, 128, device=dev) * 0.1
    bad = rows // 2 if rows > 1 else None
    if bad is not None:
        z[bad, 77] = float("nan")
    out = torch.full((16, rows + 3), 7.0, device=dev)
    _lib.call("b200pf_ln_proj_heads", ptr(z), ptr(gamma), ptr(beta), ptr(w), ptr(out), rows + 3, rows, 128, 16, stream())
    torch.cuda.synchronize()
    xn = torch.nn.functional.layer_norm(z.double(), (128,), gamma.double(), beta.double(), 1e-5)
    want = w.double() @ xn.T
    mean = z.double().mean(1, keepdim=True)
    unit = (z.double().abs() + mean.abs()) * torch.rsqrt(z.double().var(1, unbiased=False, keepdim=True) + 1e-5)
    size = (w.double().abs() * gamma.double()) @ unit.T + w.double().abs() @ beta.double().abs()[:, None]
    got = out[:, :rows].double()
    keep = torch.ones(rows, dtype=torch.bool, device=dev)
    if bad is not None:
        keep[bad] = False
        assert torch.isnan(got[:, bad]).all()
    assert ((got - want).abs()[:, keep] <= 2.0 ** -19 * size[:, keep]).all()
    assert (out[:, rows:] == 7).all()
