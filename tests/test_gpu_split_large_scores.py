"""Attention of the fp32-accurate path at scores of any size.

The triangle attention as a whole with the LayerNorm gain times g: scores grow with g * g, up to where none of their bits says anything about the
probabilities; the result has to stay finite, no part may overflow.

The softmax itself on scores that are known exactly (a bias that is a multiple of the scores' ulp, queries of nearly zero): equal keys give the mean
of their values, one key far above the rest gives its own, two at a known distance share as 2^distance to one, wherever in the row they stand
(first, second or third tile of 64 keys) and however large the scores are.  Tolerance 2^-20 of the norm: 2^x to 2^-22, the parts of the probabilities
and of the result 2^-23 each, and sums of up to 33 truncated products, 2^-24 each at worst with signs that mostly cancel."""
import pytest
import torch

from tests.test_gpu_split import inputs, layer
from tests.test_gpu_split_exponent import track
from tt_boltz_b200 import _lib, ops, weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gain", [1e2, 3e3, 5e3, 1e4, 2e4, 5e4])
def test_large_scores_stay_finite(gain):
    dev, n = torch.device("cuda:0"), 130
    sd = layer(64, 4)
    sd["tri_att_start.layer_norm.weight"] = sd["tri_att_start.layer_norm.weight"] * gain
    _, z, pm, _ = inputs(n, 64)
    out = z.to(dev)
    ops.tri_att_split(out, pm.to(torch.uint8).to(dev), weights.pack_split_triatt(sd, "tri_att_start.", dev), False, ops.Scratch(dev))
    assert bool(torch.isfinite(out).all())
    assert _lib.device_status() == 0


@pytest.mark.parametrize("cs, heads", [(384, 16), (128, 4)])
@pytest.mark.parametrize("size", [1.0, 2.0 ** 10, 2.0 ** 20, 2.0 ** 24, 2.0 ** 30])
@pytest.mark.parametrize("at", [3, 70, 140])
def test_known_softmax_at_large_scores(cs, heads, size, at):
    dev, n, g = torch.device("cuda:0"), 150, torch.Generator().manual_seed(at)
    tr = track(cs, heads, dev)
    s = torch.stack([torch.ones(cs).index_fill(0, torch.randperm(cs, generator=g)[:cs // 2], -1.0) for _ in range(n)])
    step = max(2.0, size * 2.0 ** -22)          # a few ulps of the scores, and at least two powers of two of a probability
    other = (at + 75) % n                       # another tile's key
    bias = torch.full((heads, n, n), -size)
    kind = torch.arange(n) % 4                  # per query: all keys equal / one far above / one `step` above the rest / two keys, `step` apart, far above
    bias[:, kind == 1, at] = size * 2 + 512
    bias[:, kind == 2, at] = -size + step
    bias[:, kind == 3, at] = size * 2 + 512
    bias[:, kind == 3, other] = size * 2 + 512 - step
    p = torch.softmax(bias.double() * torch.log(torch.tensor(2.0, dtype=torch.float64)), -1)
    want = torch.einsum("hqk,khd->qhd", p, s.double().view(n, heads, -1)).reshape(n, cs)
    og = tr.attention(s.to(dev), bias.to(dev), torch.ones(n, dtype=torch.uint8, device=dev), 0, n, ops.Scratch(dev))
    got = og.double().sum(0).cpu()
    one = got[kind == 1] / s[at].double()       # the value of a key as it comes out: the scale of the parts, one half, the LayerNorm's epsilon
    scale = float(one.mean())
    assert float((one / scale - 1).abs().max()) < 2.0 ** -20
    for q in range(4):
        err, norm = (got[kind == q] / scale - want[kind == q]).norm(), want[kind == q].norm()
        assert float(err / norm) < 2.0 ** -20, q
    assert _lib.device_status() == 0
