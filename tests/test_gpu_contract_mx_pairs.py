"""The block-scaled contraction on CTA pairs against its one-CTA form, which an output in groups of one row selects: the same products in the
same order of k, so the same bits, padding columns included.  One row past a tile, one short of two, ragged k (a last block of 1 and of 127),
unequal numbers of rows on the two sides, row groups of 32 that a tile's end splits, and more tiles than there are pairs."""
import ctypes as C

import pytest
import torch

from tt_boltz_b200 import _lib
from tt_boltz_b200._lib import Planes, call, ptr, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m, n, k, channels, group", [(129, 129, 129, 3, 0), (255, 130, 255, 2, 0), (256, 512, 128, 2, 0), (257, 300, 1025, 2, 0),
                                                      (288, 288, 288, 3, 32), (640, 40, 200, 2, 320), (400, 400, 400, 80, 0)])
def test_pairs_have_the_bits_of_one_cta(m, n, k, channels, group):
    dev = "cuda:0"
    lib = _lib.load()
    g = torch.Generator(device=dev).manual_seed(m + k)
    kp, xp = (k + 15) // 16 * 16, (n + 7) // 8 * 8
    planes, scales = [], []
    for rows in (m, n):
        q = (torch.randn(channels, rows, kp, generator=g, device=dev) * 100).clamp(-448, 448).to(torch.float8_e4m3fn)
        planes.append(q)
        scales.append(torch.randint(118, 132, (lib.b200pf_mx_scale_bytes(rows, k, channels),), generator=g, device=dev, dtype=torch.uint8))
    pa, pb = (Planes(ptr(p), rows * kp, 0, kp, rows, k, 1, 0) for p, rows in zip(planes, (m, n)))

    def run(row_group):
        per = row_group or m
        x = torch.full((m // per, channels, per, xp), 7.0, dtype=torch.bfloat16, device=dev)
        call("b200pf_trimul_contract", C.byref(pa), C.byref(pb), ptr(scales[0]), ptr(scales[1]), ptr(x), per * xp, xp, row_group, channels * per * xp, channels, 2,
             stream())
        torch.cuda.synchronize()
        return x.permute(1, 0, 2, 3).reshape(channels, m, xp)

    got, want = run(group), run(1)
    assert _lib.device_status() == 0
    assert torch.isfinite(want.float()).all() and want.float().abs().max() > 0
    assert torch.equal(got, want)
