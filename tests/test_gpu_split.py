"""The fp32-accurate path on 16-bit parts (csrc/split_*.cu) against the oracle in 64 bits, at the edges of its tiles: 128-row and
32-column GEMM tiles, 64-key attention tiles, 32-position LayerNorm tiles, K splits.

Tolerance on an update's relative 2-norm: two fp16 parts keep every factor to 2^-23 and a product leaves out at most 2^-22 (2^-21
relative per product, random), and every MMA truncates its addend to an ulp of the running sum (2^-24 of it, always towards zero); the longest sum here
takes 3 * 1536 / 16 = 288 of them, 1.7e-5 at worst.  2e-5 covers both."""
import pytest
import torch

from oracle import pairformer_oracle as orc
from tt_boltz_b200 import _lib, ops, synthetic, weights

pytestmark = pytest.mark.gpu
TOL = 2e-5


def rel_l2(x, y):
    return float((x.double().cpu() - y.double().cpu()).norm() / y.double().cpu().norm())


def layer(c, heads):
    sd = synthetic.make_weights(1, seed=3, std=0.05, affine_jitter=0.2, c_z=c, tri_heads=heads)
    return {k[len("layers.0."):]: v for k, v in sd.items()}


def inputs(n, c):
    s, z = synthetic.make_inputs(n, c_z=c, seed=n)
    g = torch.Generator().manual_seed(n)
    pm = torch.rand(n, n, generator=g) > 0.2
    pm[:, 0] = True
    pm[0, :] = True
    tm = torch.ones(n)
    tm[max(1, n - 3):] = 0
    return s[0], z[0], pm, tm


@pytest.mark.parametrize("c,heads", [(64, 4), (128, 4), (256, 8)])
@pytest.mark.parametrize("n", [1, 31, 65, 130])
def test_pair_sub_operations(c, heads, n):
    dev = torch.device("cuda:0")
    sd = layer(c, heads)
    w64 = {k: v.double() for k, v in sd.items()}
    _, z, pm, _ = inputs(n, c)
    pm_u8, scratch = pm.to(torch.uint8).to(dev), ops.Scratch(dev)
    cases = [("tri_mul_out", lambda zz: ops.tri_mul_split(zz, pm_u8, weights.pack_split_trimul(sd, "tri_mul_out.", dev), False, scratch),
              orc.tri_mul(z.double(), w64, "tri_mul_out", pm.double(), False)),
             ("tri_mul_in", lambda zz: ops.tri_mul_split(zz, pm_u8, weights.pack_split_trimul(sd, "tri_mul_in.", dev), True, scratch),
              orc.tri_mul(z.double(), w64, "tri_mul_in", pm.double(), True)),
             ("tri_att_start", lambda zz: ops.tri_att_split(zz, pm_u8, weights.pack_split_triatt(sd, "tri_att_start.", dev), False, scratch),
              orc.tri_att(z.double(), w64, "tri_att_start", pm.double(), False)),
             ("tri_att_end", lambda zz: ops.tri_att_split(zz, pm_u8, weights.pack_split_triatt(sd, "tri_att_end.", dev), True, scratch),
              orc.tri_att(z.double(), w64, "tri_att_end", pm.double(), True)),
             ("transition", lambda zz: ops.transition_split(zz, weights.pack_split_transition(sd, "transition_z.", dev), scratch),
              orc.transition(z.double(), w64, "transition_z"))]
    for name, run, want in cases:
        zd = z.to(dev)
        before = zd.clone()
        run(zd)
        # the update is read back as a difference of fp32 values: half an ulp of z on top of the tolerance
        slack = float(2.0 ** -24 * before.double().norm() / want.norm())
        assert rel_l2(zd.double() - before.double(), want) < TOL + slack, (name, c, n)
    assert _lib.device_status() == 0


@pytest.mark.parametrize("n", [1, 63, 129, 300])
def test_single_track(n):
    """All query rows at once, and the same rows in two ranges as the sharded trunk computes them (bit-identical attention)."""
    dev = torch.device("cuda:0")
    sd = layer(128, 4)
    w64 = {k: v.double() for k, v in sd.items()}
    s, z, _, tm = inputs(n, 128)
    track = ops.pack_single_track(sd, "", 16, dev)
    assert isinstance(track, ops.SingleTrack)
    want = s.double() + orc.attention_pair_bias(orc._ln(s.double(), w64, "pre_norm_s"), z.double(), tm.double(), w64, "attention", 16)
    want = want + orc.transition(want, w64, "transition_s")
    sd_, zd, tm_u8 = s.to(dev), z.to(dev), tm.to(torch.uint8).to(dev)
    scratch = ops.Scratch(dev)
    whole = track.attention(sd_, track.bias(zd), tm_u8, 0, n, scratch)
    half = (n + 1) // 2
    parts = [track.attention(sd_, track.bias(zd[r0:r1].contiguous()), tm_u8, r0, r1 - r0, scratch) for r0, r1 in ((0, half), (half, n)) if r1 > r0]
    assert torch.equal(torch.cat(parts, 1), whole)
    out = sd_.clone()
    ops.single_track(out, zd, tm_u8, track, scratch)
    slack = float(2.0 ** -24 * s.double().norm() / (want - s.double()).norm())
    assert rel_l2(out.double() - sd_.double(), want - s.double()) < TOL + slack
    assert _lib.device_status() == 0


@pytest.mark.parametrize("rows,k,n,accumulate", [(1, 8, 4, False), (130, 40, 64, True), (300, 128, 100, False)])
def test_split_linear(rows, k, n, accumulate):
    """Unbounded inputs (three bf16 parts): entries over ten decades, ragged rows, K and N tails."""
    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, k, generator=g) * 10.0 ** torch.randint(-5, 6, (rows, 1), generator=g)
    w, b, y0 = torch.randn(n, k, generator=g), torch.randn(n, generator=g), torch.randn(rows, n, generator=g)
    y = y0.to(dev)
    ops.split_linear(x.to(dev), weights.bf16_parts(w, dev), b.to(dev), y, accumulate, ops.Scratch(dev))
    want = x.double() @ w.double().T + b.double() + (y0.double() if accumulate else 0)
    err = (y.cpu().double() - want).norm(dim=1) / want.norm(dim=1)
    assert float(err.max()) < 2e-6          # 24 bits of every factor: 2^-23 per term and rounding
    assert _lib.device_status() == 0
