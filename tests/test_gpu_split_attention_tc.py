"""The fp32-accurate triangle attention on tcgen05 (three lines per CTA, 128-query and 64-key tiles, half of a last tile of at most 32 keys)
at the edges of its tiles, rows and columns as lines, with the last CTA's lines short of three and with fewer lines than it takes, against
the oracle in 64 bits (tolerance as for the other sub-operations on part planes) and against the un-fused fp32 kernels, also with lines
whose keys are all masked, whose scores fp32 rounds to one value.  At most 64 keys are one tile, which the issuer handles in another order:
with 8 and 16 heads a CTA has two and more such items.  A NaN or an infinity in z stays in what it has a say in."""
import pytest
import torch

from oracle import pairformer_oracle as orc
from tests.test_gpu_split import TOL, inputs, layer, rel_l2
from tt_boltz_b200 import _lib, ops, weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ending", [False, True])
@pytest.mark.parametrize("c, heads, n", [(64, 4, n) for n in (1, 2, 3, 4, 5, 32, 33, 63, 64, 96, 97, 128, 129, 161, 200)] + [(128, 8, 67), (256, 16, 100),
                                            (256, 8, 57), (256, 8, 64), (256, 16, 50), (256, 16, 64), (64, 4, 110), (64, 4, 120)])
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


@pytest.mark.parametrize("ending", [False, True])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("n", [64, 100, 161])
def test_not_a_number_stays_in_its_line(n, value, ending):
    """One entry z[i][j] that is no number (i the line, in either form): key j of line i, and the bias between query i and key j of every
    line, where a mask does not take it away.  Line i and every line's query i are NaN then; the rest keeps its bits."""
    dev, pre, c, heads = torch.device("cuda:0"), "tri_att_end" if ending else "tri_att_start", 64, 4
    sd = layer(c, heads)
    _, z, pm, _ = inputs(n, c)
    pack, pm, i, j = weights.pack_split_triatt(sd, pre + ".", dev), pm.to(torch.uint8).to(dev), n // 2, n - 2

    def run(x):
        x = x.to(dev)
        ops.tri_att_split(x, pm, pack, ending, ops.Scratch(dev))
        assert _lib.device_status() == 0
        return x.transpose(0, 1) if ending else x
    want = run(z.clone())
    bad = z.clone()
    (bad.transpose(0, 1) if ending else bad)[i, j, 5] = value
    got = run(bad)
    touched = torch.zeros(n, n, dtype=torch.bool, device=dev)
    touched[i] = touched[:, i] = True
    assert bool(torch.isnan(got[touched]).all())
    assert torch.equal(got[~touched], want[~touched])
