"""GEMMs of the fp32-accurate path on CTA pairs, at sizes where they run on them: rows that end in either CTA's half of a tile or leave the
second one empty, an even and an odd number of 128-row tiles, columns that end inside a tile, K with a tail, in every epilogue that the pair
track has (operand planes and contraction, gated output, transition), against the oracle in 64 bits.  Tolerance as for the other
sub-operations on part planes."""
import pytest
import torch

from oracle import pairformer_oracle as orc
from tests.test_gpu_split import TOL, inputs, layer, rel_l2
from tt_boltz_b200 import _lib, ops, weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c, heads, n", [(256, 8, 97), (256, 8, 112), (256, 8, 182), (128, 4, 150), (128, 4, 257), (64, 4, 200)])
def test_pair_track(c, heads, n):
    dev = torch.device("cuda:0")
    sd = layer(c, heads)
    w64 = {k: v.double().to(dev) for k, v in sd.items()}
    _, z, pm, _ = inputs(n, c)
    z64, pm64, pm_u8, scratch = z.double().to(dev), pm.double().to(dev), pm.to(torch.uint8).to(dev), ops.Scratch(dev)
    for name in ("tri_mul_out", "tri_mul_in", "transition"):
        got = z.to(dev)
        if name == "transition":
            ops.transition_split(got, weights.pack_split_transition(sd, "transition_z.", dev), scratch)
            want = orc.transition(z64, w64, "transition_z")
        else:
            ops.tri_mul_split(got, pm_u8, weights.pack_split_trimul(sd, name + ".", dev), name == "tri_mul_in", scratch)
            want = orc.tri_mul(z64, w64, name, pm64, name == "tri_mul_in")
        slack = float(2.0 ** -24 * z64.norm() / want.norm())
        assert rel_l2(got.double() - z64, want) < TOL + slack, name
    assert _lib.device_status() == 0
