"""The MSA row kernels that stand between GEMMs as kernels of their own (the MSA modules run one kernel per stage instead) against torch
in 64 bits, at ragged token counts.  Results are one fp32 computation rounded to bf16 once: 2^-9 relative per value (4e-3 with the
largest entry's neighbours), 1e-5 where terms of order one cancel; the grouped GEMM's sums take four MMAs, each truncating a sum of up
to 50 to its ulp: 4 * 50 * 2^-23 = 2.4e-5."""
import ctypes as C

import pytest
import torch
import torch.nn.functional as F

from tt_boltz_b200._lib import Planes, call, device_status, ptr, stream

pytestmark = pytest.mark.gpu
SIZES = [(1, 1), (3, 7), (2, 64), (5, 65), (37, 130)]


def _g(s, n):
    return torch.Generator().manual_seed(100 * s + n)


def _close(got, want, slack=1e-5):
    assert torch.isfinite(got).all()
    assert bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + slack).all())


@pytest.mark.parametrize("s, n", SIZES)
def test_layernorm_rows(s, n):
    g, np_ = _g(s, n), (n + 7) // 8 * 8
    m, gam, bet = torch.randn(s, n, 64, generator=g).cuda() * 2 + 0.3, torch.randn(64, generator=g).cuda(), torch.randn(64, generator=g).cuda()
    out = torch.full((s, np_, 64), 7.0, dtype=torch.bfloat16, device="cuda")
    call("b200pf_msa_ln_bf16", ptr(m), ptr(gam), ptr(bet), ptr(out), s, n, np_, stream())
    _close(out[:, :n], F.layer_norm(m.double(), (64,), gam.double(), bet.double(), 1e-5))
    assert bool((out[:, n:] == 0).all())


@pytest.mark.parametrize("s, n", SIZES)
def test_gate_and_transpose(s, n):
    g, np_ = _g(s, n), (n + 7) // 8 * 8
    o, gate = (torch.randn(8, s, 32, np_, generator=g).bfloat16().cuda() for _ in range(2))
    val = torch.full((s, np_, 256), 7.0, dtype=torch.bfloat16, device="cuda")
    call("b200pf_pwa_gate_transpose", ptr(o), ptr(gate), ptr(val), s, np_, stream())
    _close(val, (o.double() * torch.sigmoid(gate.double())).permute(1, 3, 0, 2).reshape(s, np_, 256))


@pytest.mark.parametrize("rows", [1, 7, 8, 9, 4097])
def test_swiglu(rows):
    h = torch.randn(rows, 512, generator=_g(rows, 0)).bfloat16().cuda() * 2
    out = torch.empty(rows, 256, dtype=torch.bfloat16, device="cuda")
    call("b200pf_msa_swiglu", ptr(h), ptr(out), rows, stream())
    _close(out, F.silu(h[:, :256].double()) * h[:, 256:].double())


@pytest.mark.parametrize("s, n", SIZES)
def test_add_rows(s, n):
    g, np_ = _g(s, n), (n + 7) // 8 * 8
    m, t = torch.randn(s, n, 64, generator=g).cuda(), torch.randn(s, np_, 64, generator=g).bfloat16().cuda()
    want = m + t[:, :n].float()
    call("b200pf_msa_add_rows", ptr(m), ptr(t), s, n, np_, stream())
    assert torch.equal(m, want)


@pytest.mark.parametrize("s, n", [(1, 32), (3, 40), (5, 130)])
def test_grouped_gemm(s, n):
    """[16 heads][S][32][np] = W[512][64] x rows[S * np][64]^T, rows in groups of 32, columns in groups of np."""
    g, np_ = _g(s, n), (n + 31) // 32 * 32
    w, rows = torch.randn(512, 64, generator=g).bfloat16().cuda(), torch.randn(s * np_, 64, generator=g).bfloat16().cuda()
    out = torch.empty(16, s, 32, np_, dtype=torch.bfloat16, device="cuda")
    pa, pb = Planes(ptr(w), 512 * 64, 0, 64, 512, 64, 1, 0), Planes(ptr(rows), s * np_ * 64, 0, 64, s * np_, 64, 1, 0)
    call("b200pf_gemm_grouped", C.byref(pa), C.byref(pb), ptr(out), 0, np_, 32, s * 32 * np_, np_, 32 * np_, 1, stream())
    want = (w.double() @ rows.double().T).view(16, 32, s, np_).permute(0, 2, 1, 3)
    _close(out, want, 2.4e-5)
    assert device_status() == 0
