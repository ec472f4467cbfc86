"""The gates of the fp32-accurate GEMM's epilogues where they saturate and where they must not hide a NaN.  With the LayerNorm gain times g the
gates' arguments have a spread of A = g * sqrt(C) * 0.05 (the weights' spread): their sigmoids run from 0 to 1.  Tolerance as in
test_gpu_split, and for the arguments' own error: 2^-21 of an argument's size, A * 2^-21, times the slope, at most 1/4, in the share of some
4 / A of them that lies where the sigmoid bends: A * 2^-23 * sqrt(4 / A) = sqrt(A) * 2^-22 of the gates' norm, times 4 for what multiplies them."""
import pytest
import torch

from oracle import pairformer_oracle as orc
from tests.test_gpu_split import TOL, inputs, layer, rel_l2
from tt_boltz_b200 import _lib, ops, weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c, heads, n", [(64, 4, 33), (64, 4, 130), (256, 8, 70)])
@pytest.mark.parametrize("gain", [1e-3, 1.0, 30.0, 1e4])
def test_saturated_gates(c, heads, n, gain):
    dev = torch.device("cuda:0")
    sd = layer(c, heads)
    for name in ("transition_z.norm", "tri_mul_out.norm_in"):
        sd[name + ".weight"] = sd[name + ".weight"] * gain
    w64 = {k: v.double() for k, v in sd.items()}
    _, z, pm, _ = inputs(n, c)
    scratch, zd = ops.Scratch(dev), z.to(dev)
    for run, want in ((lambda t: ops.transition_split(t, weights.pack_split_transition(sd, "transition_z.", dev), scratch), orc.transition(z.double(), w64, "transition_z")),
                      (lambda t: ops.tri_mul_split(t, pm.to(torch.uint8).to(dev), weights.pack_split_trimul(sd, "tri_mul_out.", dev), False, scratch),
                       orc.tri_mul(z.double(), w64, "tri_mul_out", pm.double(), False))):
        out = zd.clone()
        run(out)
        slack = float(2.0 ** -24 * zd.double().norm() / want.norm())
        assert rel_l2(out.double() - zd.double(), want) < TOL + slack + (gain * c ** 0.5 * 0.05) ** 0.5 * 2.0 ** -20, gain
    assert _lib.device_status() == 0


def test_a_nan_row_stays_one():
    dev = torch.device("cuda:0")
    x = torch.randn(50, 64).to(dev)
    x[7, 3] = float("nan")
    ops.transition_split(x, weights.pack_split_transition(layer(64, 4), "transition_z.", dev), ops.Scratch(dev))
    assert bool(torch.isnan(x[7]).all()) and int(torch.isnan(x).any(1).sum()) == 1
