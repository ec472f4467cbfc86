"""A single line's attention with its key tiles over three groups of warps, against 64 bits: from the first length that takes it (two tiles and
one key: two groups with a tile, one with a key) over lengths that leave the groups unequal numbers of tiles, up to the last one; lengths a
multiple of four and not (whole and single bias values); keys masked out so that a whole group's tiles hold none
that attends, or a line one that does (with none, the scores lie at 1e6, where a last place of fp32 is 2^-4).  A
range of the queries has the bits of all of them, also beyond the last length.  Tolerance: every factor (normalised row, weight, q, k, v,
probability) is held to 2^-22 and the tensor core truncates some 2^3 sums of a product to 2^-23 of their size: 2^-19 for what enters linearly.
An error of a logit is a relative one of its probabilities: 2^-20 of sum |q||k| / sqrt(24), at its root mean square, for two factors at
2^-21 each (their own parts and those of the projection that made them)."""
import pytest
import torch

from tt_boltz_b200 import _lib, ops, synthetic

pytestmark = pytest.mark.gpu
HEADS, HD = 16, 24


def reference(sd, s, bias, mask):
    n = s.shape[0]
    x = torch.nn.functional.layer_norm(s.double(), (HEADS * HD,), sd["pre_norm_s.weight"].double(), sd["pre_norm_s.bias"].double(), 1e-5)
    proj = lambda name, b=None: (x @ sd[f"attention.{name}.weight"].double().T + (0 if b is None else sd[b].double())).view(n, HEADS, HD).transpose(0, 1)
    q, k, v, gate = proj("proj_q", "attention.proj_q.bias"), proj("proj_k"), proj("proj_v"), torch.sigmoid(proj("proj_g"))
    logits = q @ k.transpose(1, 2) / HD ** 0.5 + bias.double().view(HEADS, n, n) / 1.4426950408889634 + (mask.double() - 1) * 1e6
    return ((logits.softmax(-1) @ v) * gate).transpose(0, 1).reshape(n, HEADS * HD), ((q.abs() @ k.abs().transpose(1, 2)) / HD ** 0.5).square().mean().sqrt()


def layer0(seed):
    return {k[len("layers.0."):]: v for k, v in synthetic.make_weights(1, seed=seed, std=0.1, affine_jitter=0.2, with_s=True).items() if k.startswith("layers.0.")}


@pytest.mark.parametrize("n, out", [(200, (64, 128)), (200, (0, 64)), (200, (1, 200)), (200, (0, 192)), (129, (0, 128)), (509, (64, 320)), (1025, (64, 1024))])
def test_keys_excluded_by_the_bias(n, out):
    """A bias of -inf at whole tiles of keys, a whole key group's among them, and at all keys but one: the others' softmax."""
    dev, sd = torch.device("cuda:0"), layer0(n)
    track = ops.pack_single_track(sd, "", HEADS, dev)
    g = torch.Generator().manual_seed(n)
    s, bias, mask = torch.randn(n, HEADS * HD, generator=g), torch.randn(HEADS, n, n, generator=g), torch.ones(n, dtype=torch.uint8)
    bias[:, :, out[0]:out[1]] = -float("inf")
    got = track.attention(s.to(dev), bias.view(HEADS, n * n).to(dev), mask.to(dev), 0, n, ops.Scratch(dev)).double().sum(0).cpu() / track.pack.struct.o_scale
    assert _lib.device_status() == 0
    want, size = reference(sd, s, bias, mask)
    err = (got - want).norm() / want.norm()
    assert err < 2.0 ** -19 + 2.0 ** -20 * size, (err, size)


@pytest.mark.parametrize("n, dead", [(129, None), (192, (64, 128)), (193, None), (257, (0, 192)), (320, None), (509, (64, 509)), (512, (0, 511)),
                                     (1023, None), (1024, (128, 1000)), (1025, None)])
def test_against_64_bits(n, dead):
    dev = torch.device("cuda:0")
    sd = layer0(n)
    track = ops.pack_single_track(sd, "", HEADS, dev)
    g = torch.Generator().manual_seed(n)
    s = torch.randn(n, HEADS * HD, generator=g)
    bias = torch.randn(HEADS, n * n, generator=g) * 2
    mask = torch.ones(n, dtype=torch.uint8)
    if dead is not None:
        mask[dead[0]:dead[1]] = 0
    scratch = ops.Scratch(dev)
    sg, bg, mg = s.to(dev), bias.to(dev), mask.to(dev)
    out = track.attention(sg, bg, mg, 0, n, scratch)
    for r0, r1 in ((0, 1), (n // 3, n)):
        part = track.attention(sg, bg.view(HEADS, n, n)[:, r0:r1].contiguous(), mg, r0, r1 - r0, scratch)
        assert torch.equal(part, out[:, r0:r1])
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    want, size = reference(sd, s, bias, mask)
    got = out.double().sum(0).cpu() / track.pack.struct.o_scale
    err = (got - want).norm() / want.norm()
    assert err < 2.0 ** -19 + 2.0 ** -20 * size, (err, size)
