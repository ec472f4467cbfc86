"""The un-fused fp32 kernels: the path of the fp32 tier at widths the part-plane kernels are not built for (pair width 96 with three
heads, single track of 192), and, with the part planes switched off, at the widths they have taken over.  Against the CPU oracle at that
tier's tolerance (1e-4 relative L2 per block)."""
import pytest
import torch

from oracle import pairformer_oracle as orc
from tests.conftest import rel_l2
from tt_boltz_b200 import B200PairformerModule, B200PairUpdateBlock, _lib, ops, synthetic, weights

pytestmark = pytest.mark.gpu
TOL = 1e-4


@pytest.mark.parametrize("c_z, tri_heads, c_s, heads", [(96, 3, 192, 8), (64, 4, 384, 16), (128, 4, 384, 16), (256, 8, 384, 16)])
@pytest.mark.parametrize("n", [1, 37, 65])
def test_block(c_z, tri_heads, c_s, heads, n, monkeypatch):
    monkeypatch.setattr(weights, "SPLIT_WIDTHS", ())
    sd = synthetic.make_weights(1, seed=3, std=0.04, affine_jitter=0.2, c_s=c_s, c_z=c_z, num_heads=heads, tri_heads=tri_heads)
    s, z = synthetic.make_inputs(n, c_s=c_s, c_z=c_z, seed=5)
    m, pm = synthetic.tail_padding_mask(n, n // 9)
    mod = B200PairformerModule(c_s, c_z, 1, num_heads=heads, pairwise_num_heads=tri_heads, precision="fp32")
    mod.load_state_dict(sd, strict=True)
    s_o, z_o = mod.cuda()(s.cuda(), z.cuda(), m.cuda(), pm.cuda())
    layer = mod.layers[0]
    assert not layer.split and isinstance(layer._packed["single"], ops.SingleTrackF32)
    with torch.no_grad():
        s_w, z_w = orc.pairformer_stack(s[0], z[0], m[0], pm[0], sd, 1, num_heads=heads)
    assert _lib.device_status() == 0
    assert rel_l2(z_o[0].cpu(), z_w) < TOL
    assert rel_l2(s_o[0].cpu(), s_w) < TOL


@pytest.mark.parametrize("c, hidden", [(96, 200), (256, 512)])
def test_pair_update_block(c, hidden, monkeypatch):
    monkeypatch.setattr(weights, "SPLIT_WIDTHS", ())
    n = 33
    blk = B200PairUpdateBlock(c, hidden)
    assert not blk.split
    g = torch.Generator().manual_seed(3)
    with torch.no_grad():
        for p in blk.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (0.04 if p.dim() == 2 else 0.2))
            if p.dim() == 1:
                p.add_(0.8)
    sd = blk.state_dict()
    _, z = synthetic.make_inputs(n, c_z=c, seed=8, with_s=False)
    _, pm = synthetic.tail_padding_mask(n, 2)
    with torch.no_grad():
        want = z[0] + orc.tri_mul(z[0], sd, "tri_mul_out", pm[0], False)
        want = want + orc.tri_mul(want, sd, "tri_mul_in", pm[0], True)
        want = want + orc.transition(want, sd, "transition_z")
    got = blk.cuda()(z.cuda(), pm.cuda())
    assert _lib.device_status() == 0
    assert rel_l2(got[0].cpu(), want) < TOL
