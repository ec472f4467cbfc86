"""The triangle-multiplication epilogue's LayerNorm over the channels of x, whose statistics come from the tile in shared memory: at the
edges of the 128-position tiles, with one tile per CTA and with several in turn, and with means far from zero.  The gate's weights are zero,
so the update is p' = rstd (W x - mean wsum) + wb alone.  bf16 factors are exact; sums of 128 terms in fp32 (statistics, and products that
the tensor core adds by truncation) are off by at most 128 ulps of the sum of their magnitudes, 2^-16 of it; the variance E[x^2] - mean^2
loses as much of E[x^2]."""
import pytest
import torch

from tt_boltz_b200 import _lib
from tt_boltz_b200._lib import call, ptr, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows, n", [(1, 1), (2, 33), (3, 127), (1, 128), (5, 129), (150, 130), (300, 250), (203, 203)])
def test_statistics_of_x(rows, n):
    dev, g = torch.device("cuda:0"), torch.Generator().manual_seed(1000 * rows + n)
    pitch = (n + 7) // 8 * 8
    x = torch.full((128, rows, pitch), 9.0, dtype=torch.bfloat16, device=dev)
    x[:, :, :n] = (torch.randn(128, rows, n, generator=g) * torch.rand(1, rows, n, generator=g).add(0.1) + torch.randn(1, rows, n, generator=g)).bfloat16().to(dev)
    wp = (torch.randn(128, 128, generator=g) * 0.1).bfloat16().to(dev)
    zero = torch.zeros(128, 128, dtype=torch.bfloat16, device=dev)
    wsum, wb = wp.double().sum(1).float(), torch.randn(128, generator=g).to(dev)
    one, off = torch.ones(128, device=dev), torch.zeros(128, device=dev)
    z = torch.zeros(rows, n, 128, device=dev)
    call("b200pf_trimul_epilogue_tc", ptr(z), ptr(x), rows * pitch, pitch, ptr(one), ptr(off), ptr(wp), ptr(zero), ptr(wsum), ptr(wb), rows, n, stream())
    assert _lib.device_status() == 0
    xd = x[:, :, :n].double().permute(1, 2, 0)
    mean, sq = xd.mean(-1, keepdim=True), (xd * xd).mean(-1, keepdim=True)
    var = sq - mean * mean
    rstd = (var + 1e-5).rsqrt()
    acc = xd @ wp.double().t()
    want = rstd * (acc - mean * wsum.double()) + wb.double()
    size = xd.abs() @ wp.double().abs().t() + mean.abs() * wsum.double().abs()
    bound = 2.0 ** -16 * (rstd * size + (want - wb.double()).abs() * rstd ** 2 * sq + want.abs() + wb.double().abs())
    assert bool(((z.double() - want).abs() <= bound).all())
