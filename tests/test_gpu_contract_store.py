"""The contraction's stores at the edges of their boxes (32 rows, 64 columns through a staging tile): row groups that 32 divides (staged) and that it
does not or that are not full at the end (direct stores), last boxes that only just begin, pitches beyond the columns, several tiles per CTA in
turn through the same staging tiles, on lone CTAs (up to 128 rows) and on pairs.  The planes and groups lie apart inside a larger buffer, and
everything around them has to stay as it was.  The result is an fp32 sum rounded to bf16 once: 2^-9 of a value, and 2^-24 * sqrt(K) * K < 1e-4
of order-one terms for what cancels."""
import ctypes as C

import pytest
import torch

from tt_boltz_b200 import _lib
from tt_boltz_b200._lib import Planes, call, ptr, stream

pytestmark = pytest.mark.gpu
TILE_COLS = 256          # a tile writes its columns up to the pitch, those behind the last operand row as zeros


@pytest.mark.parametrize("rows, cols, k, channels, group, extra", [(1, 1, 8, 1, 0, 0), (33, 65, 40, 3, 0, 8), (128, 257, 64, 2, 0, 0), (129, 200, 72, 2, 0, 72),
                                                                   (256, 130, 64, 3, 64, 0), (384, 64, 128, 2, 96, 8), (200, 70, 64, 2, 40, 0),
                                                                   (300, 90, 64, 2, 128, 0), (520, 513, 136, 2, 0, 7 * 8),
                                                                   (100, 300, 64, 200, 0, 0), (300, 300, 64, 100, 0, 8), (192, 70, 64, 240, 32, 200)])
def test_contract_output(rows, cols, k, channels, group, extra):
    g = torch.Generator().manual_seed(rows + cols)
    a, b = (torch.randn(channels, r, k, generator=g).bfloat16().cuda() for r in (rows, cols))
    pitch = (cols + 7) // 8 * 8 + extra
    grp = group or rows
    groups = -(-rows // grp)
    plane, lead = grp * pitch + 24, 64
    between = channels * plane + 40
    buf = torch.full((2 * lead + groups * between,), 7.0, dtype=torch.bfloat16, device="cuda")
    pa, pb = Planes(ptr(a), rows * k, 0, k, rows, k, 1, 0), Planes(ptr(b), cols * k, 0, k, cols, k, 1, 0)
    call("b200pf_trimul_contract", C.byref(pa), C.byref(pb), None, None, ptr(buf[lead:]), plane, pitch, group, between, channels, 0, stream())
    want = torch.einsum("dik,djk->dij", a.double(), b.double())
    written = torch.zeros_like(buf, dtype=torch.bool)
    shape = (groups, channels, grp, pitch), (between, plane, pitch, 1), lead
    rows_of = lambda t: t.as_strided(*shape).permute(0, 2, 1, 3).reshape(groups * grp, channels, pitch)[:rows].transpose(0, 1)
    got = rows_of(buf).double()
    assert bool(((got[..., :cols] - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all())
    last = min(pitch, -(-cols // TILE_COLS) * TILE_COLS)
    assert bool((got[..., cols:last] == 0).all())
    for r in range(rows):
        written.as_strided(*shape)[r // grp, :, r % grp, :last] = True
    assert bool((buf[~written] == 7).all())
    assert _lib.device_status() == 0
