"""The exponent of the fp32-accurate attention.  The score of a key close to its row's maximum differs from it by little, and that difference is
exact: what the low bits of such scores say must reach the probabilities.

Queries are (nearly) zero, so the scores are the bias; values are +-1 after the LayerNorm, gates one half.  The result is compared with
64 bits up to a common factor (the LayerNorm's epsilon), once with scores on a grid of 2^-16, where no arithmetic on them rounds, and once
with the same scores off the grid.  The scores, below 2 in size, come with an ulp of 2^-23 and their differences, below 4, round at half of 2^-22:
7e-8 of a probability at most and a third of that in the norm, beside an error of some 1.7e-7 (2^x to some 2^-22, the parts, the sums), so the two
errors differ by some 2 %.  An exponent that carries a constant of 8 to 16 as well rounds at 2^-20: 1.9e-7 in the norm, half as much
again."""
import math

import pytest
import torch

from tt_boltz_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def track(cs, heads, dev):
    one, zero, eye = torch.ones(cs), torch.zeros(cs), torch.eye(cs)
    sd = {"pre_norm_s.weight": one, "pre_norm_s.bias": zero, "transition_s.norm.weight": one, "transition_s.norm.bias": zero,
          "attention.proj_q.weight": eye * 1e-12, "attention.proj_q.bias": zero, "attention.proj_k.weight": eye, "attention.proj_v.weight": eye,
          "attention.proj_g.weight": torch.zeros(cs, cs), "attention.proj_o.weight": eye, "attention.proj_z.0.weight": torch.ones(128),
          "attention.proj_z.0.bias": torch.zeros(128), "attention.proj_z.1.weight": torch.zeros(heads, 128),
          "transition_s.fc1.weight": torch.ones(64, cs), "transition_s.fc2.weight": torch.ones(64, cs), "transition_s.fc3.weight": torch.ones(cs, 64)}
    return ops.SingleTrack({"x." + k: v for k, v in sd.items()}, "x.", heads, dev)


def error(tr, s, bias, dev):
    """Relative 2-norm of the attention's own error; s [n, cs] of +-1 with mean zero, bias [heads, n, n] in base-2 logarithms."""
    n, cs = s.shape
    og = tr.attention(s.to(dev), bias.to(dev), torch.ones(n, dtype=torch.uint8, device=dev), 0, n, ops.Scratch(dev))
    got = og.double().sum(0).cpu()
    p = torch.softmax(bias.double() * math.log(2.0), -1)
    want = torch.einsum("hqk,khd->qhd", p, s.double().view(n, len(bias), -1)).reshape(n, cs)
    want = want * ((got * want).sum() / (want * want).sum())
    return float((got - want).norm() / want.norm())


@pytest.mark.parametrize("n, cs, heads", [(65, 384, 16), (292, 384, 16), (292, 128, 4)])
@pytest.mark.parametrize("spread", [0.05, 0.25])
def test_low_bits_of_scores(n, cs, heads, spread):
    dev, g = torch.device("cuda:0"), torch.Generator().manual_seed(n)
    tr = track(cs, heads, dev)
    s = torch.stack([torch.ones(cs).index_fill(0, torch.randperm(cs, generator=g)[:cs // 2], -1.0) for _ in range(n)])
    bias = (torch.randn(heads, n, n, generator=g) * spread).clamp(-1.9, 1.9)
    on_grid = (bias * 2 ** 16).round() / 2 ** 16
    e, e_grid = error(tr, s, bias, dev), error(tr, s, on_grid, dev)
    print(f"n {n} heads {heads} spread {spread}: {e:.3e}, on the grid {e_grid:.3e}")
    assert e < 1.15 * e_grid
    assert _lib.device_status() == 0
