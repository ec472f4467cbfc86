"""The contraction's staged stores at the edges of their boxes (32 rows, 64 columns; 32 in the block-scaled kernel): row groups that 32 divides and
that it does not, last boxes that only just begin, pitches beyond the columns, and memory around the output that must stay as it was.  The result
is an fp32 sum rounded to bf16 once: 2^-9 of a value, and 2^-24 * sqrt(K) * K < 1e-4 of order-one terms for what cancels."""
import ctypes as C

import pytest
import torch

from tt_boltz_b200 import _lib
from tt_boltz_b200._lib import Planes, call, ptr, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows, cols, k, channels, group, extra", [(1, 1, 8, 1, 0, 0), (33, 65, 40, 3, 0, 8), (128, 257, 64, 2, 0, 0), (129, 200, 72, 2, 0, 72),
                                                                   (256, 130, 64, 3, 64, 0), (384, 64, 128, 2, 96, 8), (200, 70, 64, 2, 40, 0),
                                                                   (300, 90, 64, 2, 128, 0), (520, 513, 136, 2, 0, 7 * 8)])
def test_contract_output(rows, cols, k, channels, group, extra):
    g = torch.Generator().manual_seed(rows + cols)
    a, b = (torch.randn(channels, r, k, generator=g).bfloat16().cuda() for r in (rows, cols))
    pitch = (cols + 7) // 8 * 8 + extra
    grp = group or rows
    groups = -(-rows // grp)
    x = torch.full((groups, channels, grp, pitch), 7.0, dtype=torch.bfloat16, device="cuda")
    pa, pb = Planes(ptr(a), rows * k, 0, k, rows, k, 1, 0), Planes(ptr(b), cols * k, 0, k, cols, k, 1, 0)
    call("b200pf_trimul_contract", C.byref(pa), C.byref(pb), None, None, ptr(x), grp * pitch, pitch, group, channels * grp * pitch, channels, 0, stream())
    want = torch.einsum("dik,djk->dij", a.double(), b.double())
    got = x.permute(1, 0, 2, 3).reshape(channels, groups * grp, pitch).double()
    assert bool(((got[:, :rows, :cols] - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all())
    assert bool((got[:, rows:] == 7).all())                                # rows of a last group that is not full are not written
    assert _lib.device_status() == 0
