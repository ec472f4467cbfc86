"""The fp32-accurate triangle attention on tcgen05 (three lines per CTA, 128-query and 64-key tiles, half of a last tile of at most 32 keys)
at the edges of its tiles, rows and columns as lines, with the last CTA's lines short of three and with fewer lines than it takes, against
the oracle in 64 bits (tolerance as for the other sub-operations on part planes) and against the un-fused fp32 kernels, also with lines
whose keys are all masked, whose scores fp32 rounds to one value."""
import pytest
import torch

from oracle import pairformer_oracle as orc
from tests.test_gpu_split import TOL, inputs, layer, rel_l2
from tt_boltz_b200 import _lib, ops, weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ending", [False, True])
@pytest.mark.parametrize("c, heads, n", [(64, 4, n) for n in (1, 2, 3, 4, 5, 32, 33, 63, 64, 96, 97, 128, 129, 161, 200)] + [(128, 8, 67), (256, 16, 100)])
def test_triangle_attention(c, heads, n, ending):
    dev, pre = torch.device("cuda:0"), "tri_att_end" if ending else "tri_att_start"
    sd = layer(c, heads)
    _, z, pm, _ = inputs(n, c)
    pack = weights.pack_split_triatt(sd, pre + ".", dev)

    def update(mask):
        zd = z.to(dev)
        ops.tri_att_split(zd, mask.to(torch.uint8).to(dev), pack, ending, ops.Scratch(dev))
        assert _lib.device_status() == 0
        return zd.double().cpu() - z.double()
    want = orc.tri_att(z.double(), {k: v.double() for k, v in sd.items()}, pre, pm.double(), ending)
    slack = float(2.0 ** -24 * z.double().norm() / want.norm())
    assert rel_l2(update(pm), want) < TOL + slack
    pm[n // 2, :] = False
    pm[:, n // 3] = False
    other = z.to(dev)
    ops.tri_att_f32(other, pm.to(torch.uint8).to(dev), weights.to_device_f32(sd, pre + ".", dev), ending)
    got, other = update(pm), other.double().cpu() - z.double()
    assert rel_l2(got, other) < TOL + 2 * slack
