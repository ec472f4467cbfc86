"""The q | k | v | gate GEMM of the fp32-accurate path at sizes where a CTA stores a gate tile (fp32, both slots of a warp's staging)
and then a q, k or v tile (16-bit parts, slot by slot): three to seven column tiles over 148 CTAs.  A store that did not wait for the
one before would show as gates that differ between runs and from the oracle in 64 bits.  Tolerance as in test_gpu_split."""
import pytest
import torch

from oracle import pairformer_oracle as orc
from tests.test_gpu_split import TOL, inputs, layer, rel_l2
from tt_boltz_b200 import _lib, ops, weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c, heads, n", [(64, 4, 98), (64, 4, 105), (64, 4, 112), (128, 4, 100), (256, 8, 69), (256, 8, 80), (256, 8, 86), (256, 8, 100),
                                         (256, 8, 121)])
def test_gate_tile_before_part_tile(c, heads, n):
    dev = torch.device("cuda:0")
    sd = layer(c, heads)
    w64 = {k: v.double().to(dev) for k, v in sd.items()}
    _, z, pm, _ = inputs(n, c)
    zd, pmd = z.to(dev), pm.to(dev)
    pm_u8, scratch = pmd.to(torch.uint8), ops.Scratch(dev)
    for pre, ending in (("tri_att_start", False), ("tri_att_end", True)):
        pack = weights.pack_split_triatt(sd, pre + ".", dev)
        outs = []
        for _ in range(8):
            out = zd.clone()
            ops.tri_att_split(out, pm_u8, pack, ending, scratch)
            outs.append(out)
        assert all(torch.equal(o, outs[0]) for o in outs[1:])
        with dev:                                   # the oracle on the GPU: new tensors there too
            want = orc.tri_att(zd.double(), w64, pre, pmd.double(), ending)
        slack = float(2.0 ** -24 * zd.double().norm() / want.norm())
        assert rel_l2(outs[0].double() - zd.double(), want) < TOL + slack
    assert _lib.device_status() == 0


@pytest.mark.parametrize("n", [3073, 3100])
def test_gate_tile_before_part_tile_in_the_single_track(n):
    dev, heads, hd = torch.device("cuda:0"), 16, 24
    sd = layer(128, 4)
    track = ops.pack_single_track(sd, "", heads, dev)
    s = inputs(4, 128)[0].new_empty(n, heads * hd).normal_(generator=torch.Generator().manual_seed(n)).to(dev)
    bias, scratch = torch.zeros(heads, n, n, device=dev), ops.Scratch(dev)
    outs = [track.attention(s, bias, None, 0, n, scratch) for _ in range(4)]
    assert all(torch.equal(o, outs[0]) for o in outs[1:])
    w = {k: v.double().to(dev) for k, v in sd.items()}
    x = orc._ln(s.double(), w, "pre_norm_s")
    lin = lambda name: (x @ w[f"attention.{name}.weight"].T)
    q, k, v = (t.view(n, heads, hd).transpose(0, 1) for t in (lin("proj_q") + w["attention.proj_q.bias"], lin("proj_k"), lin("proj_v")))
    want = torch.cat([torch.softmax(q[h] @ k[h].T / hd ** 0.5, -1) @ v[h] for h in range(heads)], 1) * torch.sigmoid(lin("proj_g"))
    got = outs[0].double().sum(0) / track.pack.struct.o_scale
    assert rel_l2(got, want) < TOL
    assert _lib.device_status() == 0
