"""Two claims that the fp32-accurate path's accuracy rests on: what two fp16 parts keep of a value (in torch, on the CPU), and on the GPU
what its attention keeps of a probability, whose exponential is the bare approximate instruction."""
import pytest
import torch


@pytest.mark.parametrize("below", range(0, 24))
def test_two_fp16_parts(below):
    """Scaled values of one binade, ``below`` binades under the largest (2^14): 2^-23 of the value, or 2^-39 of 2^14 where that is more."""
    v = (1 + torch.arange(0, 1 << 23, 7, dtype=torch.float64) * 2.0 ** -23).float() * 2.0 ** (13 - below)
    hi = v.half()
    lo = (v - hi.float()).half()
    err = (hi.double() + lo.double() - v.double()).abs()
    assert torch.isfinite(hi).all()
    assert bool((err <= torch.clamp(v.double() * 2.0 ** -23, min=2.0 ** -25)).all())


@pytest.mark.gpu
@pytest.mark.parametrize("spread", [1.0, 30.0, 400.0])
def test_attention_keeps_its_probabilities(spread):
    """Scores that are the bias alone (q = 0), one of them zero in every row and the others down to -spread in base-2 logarithms: below
    -126 the probabilities are flushed.  Per output, relative to the sum of its terms' sizes (a value counts at least its rms): 2^-22
    each for the exponentials of the probability and of the row's sum, 2^-21 for a product of parts, at most 96 / 4 + 5 additions of 2^-24
    in the row's sum and 12 MMAs of 2^-24 per tile of 64 keys (two here), 2^-21 for gate and division, 2^-19 for the values, which are a
    384-long product themselves: 7e-6 in the worst case."""
    from oracle import pairformer_oracle as orc
    from tests.test_gpu_split import inputs, layer
    from tt_boltz_b200 import _lib, ops
    dev, n, heads, hd = torch.device("cuda:0"), 96, 16, 24
    sd = layer(128, 4)
    sd["attention.proj_q.weight"] = torch.zeros_like(sd["attention.proj_q.weight"])
    sd["attention.proj_q.bias"] = torch.zeros_like(sd["attention.proj_q.bias"])
    track = ops.pack_single_track(sd, "", heads, dev)
    s = inputs(n, 128)[0].to(dev)
    g = torch.Generator().manual_seed(5)
    bias = -torch.rand(heads, n, n, generator=g) * spread
    bias[:, torch.arange(n), torch.randint(0, n, (n,), generator=g)] = 0.0
    bias = bias.to(dev)
    og = track.attention(s, bias, None, 0, n, ops.Scratch(dev))
    w = {k: v.double().to(dev) for k, v in sd.items()}
    x = orc._ln(s.double(), w, "pre_norm_s")
    v = (x @ w["attention.proj_v.weight"].T).view(n, heads, hd).transpose(0, 1)
    gate = torch.sigmoid(x @ w["attention.proj_g.weight"].T)
    p = torch.softmax(bias.double() * 0.6931471805599453, -1)
    want, size = ((p @ t).transpose(0, 1).reshape(n, heads * hd) * gate for t in (v, v.abs().clamp_min(float(v.square().mean().sqrt()))))
    got = og.double().sum(0) / track.pack.struct.o_scale
    assert float(((got - want).abs() / size).max()) < 7e-6
    assert _lib.device_status() == 0
