"""The outer product's blocks of 32 x 32 leave as bulk copies of 2 KB: one and several pairs, odd numbers of columns' tokens (half a staging
tile), at most one tile of rows (the one-CTA kernel) and more (CTA pairs), rows that end inside a tile, more tiles than there are CTAs.  Small
whole numbers: every sum is exact in fp32, so the result is the rounded one, and nothing is written behind the last pair."""
import pytest
import torch

from tt_boltz_b200 import _lib
from tt_boltz_b200._lib import call, ptr, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s_len, n_i, n_j", [(1, 1, 1), (9, 1, 3), (64, 4, 7), (65, 5, 1), (130, 9, 17), (33, 16, 16), (100, 75, 131)])
def test_blocks_are_exact(s_len, n_i, n_j):
    g = torch.Generator().manual_seed(s_len + n_j)
    pitch = (s_len + 7) // 8 * 8
    a, b = (torch.randint(-4, 5, (n, 32, pitch), generator=g).to(torch.bfloat16).cuda() for n in (n_i, n_j))
    out = torch.full((n_i * n_j + 2, 1024), 7.0, dtype=torch.bfloat16, device="cuda")
    call("b200pf_opm_outer", ptr(a), ptr(b), ptr(out), s_len, n_i, n_j, pitch, stream())
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    want = torch.einsum("ics,jds->ijcd", a[..., :s_len].double(), b[..., :s_len].double()).to(torch.bfloat16)
    assert torch.equal(out[:-2].view(n_i, n_j, 32, 32), want)
    assert (out[-2:] == 7).all()
