"""The mask of the triangle-multiplication producer: a masked position's row is zeroed before the products, so its operands are zero, and every
other position's are, to the bit, what they are without a mask.  At the edges of the tiles (128 positions of a line), with one tile per CTA and
with several in turn, whose masks the loaders fetch a tile ahead."""
import ctypes as C

import pytest
import torch

from tt_boltz_b200 import B200PairformerModule, _lib, ops, synthetic
from tt_boltz_b200._lib import PlaneOut, call, ptr, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows, n", [(1, 1), (3, 33), (130, 130), (128, 128), (203, 203), (300, 300), (64, 390), (200, 260)])
@pytest.mark.parametrize("incoming", [0, 1])
def test_masked_positions_and_no_others(rows, n, incoming):
    dev, g = torch.device("cuda:0"), torch.Generator().manual_seed(rows * 1000 + n)
    mod = B200PairformerModule(384, 128, 1, v2=True)
    mod.load_state_dict(synthetic.make_weights(1, seed=3, std=0.05, affine_jitter=0.2), strict=True)
    w = mod.layers[0]._pack(dev)["tri_mul_in" if incoming else "tri_mul_out"]
    lines, span = (n, rows) if incoming else (rows, n)
    pitch = (span + 7) // 8 * 8
    z = torch.randn(rows, n, 128, generator=g).to(dev)
    mask = (torch.rand(rows, n, generator=g) > 0.3).to(torch.uint8).to(dev)

    def planes(m):
        a, b = (torch.full((128, lines, pitch), 7.0, dtype=torch.bfloat16, device=dev) for _ in range(2))
        oa, ob = (PlaneOut(ptr(t), lines * pitch, 0, 0) for t in (a, b))
        call("b200pf_trimul_producer", ptr(z), ptr(m), *ops.trimul_producer_weights(w), C.byref(oa), C.byref(ob), pitch, rows, n, incoming, stream())
        return a[..., :span], b[..., :span]
    keep = (mask.t() if incoming else mask).bool()                          # [line][position]
    for got, free in zip(planes(mask), planes(torch.ones_like(mask))):
        assert torch.equal(got, torch.where(keep, free, torch.zeros_like(free)))
        assert bool((free != 0).any())
    assert _lib.device_status() == 0
