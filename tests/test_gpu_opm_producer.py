"""The outer-product producer (LayerNorm, both projections, mask, transposed) against torch in 64 bits at the edges of its tiles: 64
sequences a CTA and token, in two halves of eight quads, several tokens per CTA, output rows whose pitch allows no 8-byte stores.  A sum of 64
products in fp32 is off by less than 64 * 2^-24 of the largest partial sum, 1e-5 where terms of order one cancel; the result is rounded to bf16
once (2^-9)."""
import pytest
import torch
import torch.nn.functional as F

from tt_boltz_b200._lib import call, device_status, ptr, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s, n, pitch", [(1, 1, 8), (7, 3, 8), (9, 5, 9), (32, 2, 32), (33, 4, 40), (127, 3, 127), (128, 6, 128), (129, 7, 136),
                                         (260, 611, 264)])
def test_opm_producer(s, n, pitch):
    g = torch.Generator().manual_seed(s * 1000 + n)
    m, w = torch.randn(s, n, 64, generator=g).cuda() * 3 + 0.4, torch.randn(64, 64, generator=g).cuda() * 0.2
    gam, bet = torch.randn(64, generator=g).cuda(), torch.randn(64, generator=g).cuda()
    mask = (torch.rand(s, n, generator=g) > 0.2).to(torch.uint8).cuda()
    out = [torch.full((n * 32, pitch), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    call("b200pf_opm_producer", ptr(m), ptr(mask), ptr(gam), ptr(bet), ptr(w), ptr(out[0]), ptr(out[1]), s, n, pitch, stream())
    x = F.layer_norm(m.double(), (64,), gam.double(), bet.double(), 1e-5)
    want = (x @ w.double().T * mask[..., None].double()).permute(1, 2, 0)                 # [n][64][s]
    for got, ref in zip(out, (want[:, :32], want[:, 32:])):
        got, ref = got.double(), ref.reshape(n * 32, s)
        assert bool(((got[:, :s] - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5).all())
        assert bool((got[:, s:] == 7).all())                                              # nothing behind the last sequence is written
    assert device_status() == 0


def test_opm_producer_keeps_nan():
    m, mask = torch.randn(40, 2, 64).cuda(), torch.ones(40, 2, dtype=torch.uint8).cuda()
    m[3, 1, 5] = float("nan")
    w, one, zero = torch.randn(64, 64).cuda(), torch.ones(64).cuda(), torch.zeros(64).cuda()
    out = [torch.zeros(64, 40, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    call("b200pf_opm_producer", ptr(m), ptr(mask), ptr(one), ptr(zero), ptr(w), ptr(out[0]), ptr(out[1]), 40, 2, 40, stream())
    for o in out:
        bad = torch.isnan(o)
        assert bool(bad[32:, 3].all()) and int(bad.sum()) == 32


@pytest.mark.parametrize("s, n, pitch", [(1, 1, 8), (63, 5, 63), (64, 70, 64), (65, 3, 68), (190, 131, 192)])
def test_opm_producer_bits(s, n, pitch):
    """Every sum is an fp32 sum in one order, so the bf16 results are known to the bit: the channels in turn for the mean and the variance;
    for an output one chain of fused multiply-adds over channels 3 2 1 0, 11 10 9 8, .. and one over 7 6 5 4, 15 14 13 12, .., added.  A
    fused multiply-add is a product in 64 bits (exact) added and rounded; the second rounding it takes here shows once in 2^29."""
    g = torch.Generator().manual_seed(s * 1000 + n)
    m, w = torch.randn(s, n, 64, generator=g).cuda() * 3 + 0.4, torch.randn(64, 64, generator=g).cuda() * 0.2
    gam, bet = torch.randn(64, generator=g).cuda(), torch.randn(64, generator=g).cuda()
    mask = (torch.rand(s, n, generator=g) > 0.2).to(torch.uint8).cuda()
    out = [torch.full((n * 32, pitch), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    call("b200pf_opm_producer", ptr(m), ptr(mask), ptr(gam), ptr(bet), ptr(w), ptr(out[0]), ptr(out[1]), s, n, pitch, stream())
    fma = lambda a, b, c: (a.double() * b.double() + c.double()).float()
    total, ss = torch.zeros(s, n, device="cuda"), torch.zeros(s, n, device="cuda")
    for k in range(64):
        total = total + m[..., k]
    x = m - (total * (1.0 / 64))[..., None]
    for k in range(64):
        ss = fma(x[..., k], x[..., k], ss)
    x = fma(x * torch.rsqrt(ss * (1.0 / 64) + 1e-5)[..., None], gam, bet)
    chains = [torch.zeros(s, n, 64, device="cuda") for _ in range(2)]
    for k4 in range(16):
        for k in range(4 * k4 + 3, 4 * k4 - 1, -1):
            chains[k4 & 1] = fma(w[:, k], x[..., k, None], chains[k4 & 1])
    want = ((chains[0] + chains[1]) * mask[..., None]).bfloat16().permute(1, 2, 0)        # [n][64][s]
    for got, ref in zip(out, (want[:, :32], want[:, 32:])):
        assert torch.equal(got[:, :s], ref.reshape(n * 32, s))
        assert bool((got[:, s:] == 7).all())
    assert device_status() == 0
