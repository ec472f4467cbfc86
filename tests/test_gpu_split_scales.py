"""The fp32-accurate attention and triangle multiplication where their operands' scales and copies change: token counts whose bias
rows are copied in 16-byte pieces (multiples of four) and not, and weights far from the size the fp16 parts are laid out for, so that
the packed scales have to carry them.  Against the oracle in 64 bits; tolerance as in test_gpu_split (2^-21 relative per product, a
sum of truncated additions: 2e-5), plus half an ulp of z where the update is read back as a difference."""
import pytest
import torch

from oracle import pairformer_oracle as orc
from tests.test_gpu_split import TOL, inputs, layer, rel_l2
from tt_boltz_b200 import _lib, ops, weights

pytestmark = pytest.mark.gpu


def _check(run, want, z):
    zd = z.to("cuda")
    before = zd.clone()
    run(zd)
    assert torch.isfinite(zd).all() and _lib.device_status() == 0
    slack = float(2.0 ** -24 * before.double().norm() / want.norm())
    assert rel_l2(zd.double() - before.double(), want) < TOL + slack


@pytest.mark.parametrize("n", [4, 60, 64, 66, 68, 127, 128, 132, 200])
def test_bias_copies(n):
    dev, c, heads = torch.device("cuda:0"), 64, 4
    sd = layer(c, heads)
    w64 = {k: v.double() for k, v in sd.items()}
    _, z, pm, _ = inputs(n, c)
    pm_u8, scratch = pm.to(torch.uint8).to(dev), ops.Scratch(dev)
    for pre, ending in (("tri_att_start", False), ("tri_att_end", True)):
        pack = weights.pack_split_triatt(sd, pre + ".", dev)
        _check(lambda zz: ops.tri_att_split(zz, pm_u8, pack, ending, scratch), orc.tri_att(z.double(), w64, pre, pm.double(), ending), z)


@pytest.mark.parametrize("names, factor", [(("mha.linear_q.weight", "mha.linear_k.weight"), 1e-6), (("mha.linear_q.weight",), 20.0), (("mha.linear_v.weight",), 1e-3),
                                           (("mha.linear_v.weight",), 1e4), (("layer_norm.weight",), 8.0)])
def test_attention_weights_of_other_sizes(names, factor):
    dev, c, heads, n = torch.device("cuda:0"), 128, 4, 70
    sd = layer(c, heads)
    for name in names:
        sd["tri_att_start." + name] = sd["tri_att_start." + name] * factor
    w64 = {k: v.double() for k, v in sd.items()}
    _, z, pm, _ = inputs(n, c)
    pm_u8, scratch = pm.to(torch.uint8).to(dev), ops.Scratch(dev)
    pack = weights.pack_split_triatt(sd, "tri_att_start.", dev)
    _check(lambda zz: ops.tri_att_split(zz, pm_u8, pack, False, scratch), orc.tri_att(z.double(), w64, "tri_att_start", pm.double(), False), z)


@pytest.mark.parametrize("n", [4, 129])
@pytest.mark.parametrize("factor", [1.0, 1e-2, 1e3])
def test_triangle_multiplication_weights_of_other_sizes(n, factor):
    dev, c = torch.device("cuda:0"), 64
    sd = layer(c, 4)
    sd["tri_mul_out.p_in.weight"] = sd["tri_mul_out.p_in.weight"] * factor
    w64 = {k: v.double() for k, v in sd.items()}
    _, z, pm, _ = inputs(n, c)
    pm_u8, scratch = pm.to(torch.uint8).to(dev), ops.Scratch(dev)
    pack = weights.pack_split_trimul(sd, "tri_mul_out.", dev)
    _check(lambda zz: ops.tri_mul_split(zz, pm_u8, pack, False, scratch), orc.tri_mul(z.double(), w64, "tri_mul_out", pm.double(), False), z)
