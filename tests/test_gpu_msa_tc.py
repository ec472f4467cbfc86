"""The one-kernel-per-stage MSA row kernels against torch in 64 bits, at the edges of their 128-row tiles: sizes below, at and
just above a tile and its 64-token halves, several tiles per CTA, and lines that start anywhere in the tensor.

Tolerances, from the operands' 2^-9 relative rounding (bf16): the values are one product of a rounded row and a rounded weight
row, whose errors add in quadrature over the 64 channels, about 2^-9 * sqrt(2 / 3) = 1.6e-3 of the result's norm, and once more
rounded on store: 4e-3.  The updates pass two more roundings (hidden layer or gated average, second weight): 8e-3."""
import pytest
import torch
import torch.nn.functional as F

from tests.conftest import rel_l2
from tt_boltz_b200 import _lib
from tt_boltz_b200._lib import call, ptr, stream

pytestmark = pytest.mark.gpu


def _inputs(s, n, seed=0):
    g = torch.Generator().manual_seed(seed)
    m = torch.randn(s, n, 64, generator=g) * 2 + 0.3
    return g, m, torch.randn(64, generator=g) * 0.2 + 1, torch.randn(64, generator=g) * 0.2


def _w(g, rows, cols, std=0.15):
    return (torch.randn(rows, cols, generator=g) * std).bfloat16()


def _ln(m, gam, bet):
    return F.layer_norm(m.double(), (64,), gam.double(), bet.double(), 1e-5)


def _cuda(*ts):
    return [t.cuda().contiguous() for t in ts]


@pytest.mark.parametrize("rows", [1, 2, 31, 127, 128, 129, 128 * 148 + 5, 128 * 148 * 3 - 1])
def test_transition(rows):
    g, m, gam, bet = _inputs(1, rows)
    fc1, fc2, fc3 = _w(g, 256, 64), _w(g, 256, 64), _w(g, 64, 256)
    x = _ln(m, gam, bet)
    want = m.double() + (F.silu(x @ fc1.double().T) * (x @ fc2.double().T)) @ fc3.double().T
    w12 = torch.stack([fc1.view(4, 64, 64), fc2.view(4, 64, 64)], 1)
    mc, gc, bc, w12c, w3c = _cuda(m, gam, bet, w12, fc3)
    call("b200pf_msa_transition", ptr(mc), ptr(gc), ptr(bc), ptr(w12c), ptr(w3c), rows, stream())
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    assert rel_l2(mc.cpu().double() - m.double(), want - m.double()) < 8e-3


@pytest.mark.parametrize("s, n", [(1, 1), (3, 7), (5, 63), (2, 64), (2, 65), (4, 128), (300, 129), (37, 200), (160, 131)])
def test_value_and_output(s, n):
    g, m, gam, bet = _inputs(s, n, seed=1)
    w_m, w_g, w_o = _w(g, 256, 64), _w(g, 256, 64), _w(g, 64, 256)
    np_ = (n + 7) // 8 * 8
    x = _ln(m, gam, bet)
    mc, gc, bc, wm, wg, wo = _cuda(m, gam, bet, w_m, w_g, w_o)
    v = torch.full((8, s, 32, np_), 7.0, dtype=torch.bfloat16, device="cuda")
    call("b200pf_pwa_value", ptr(mc), ptr(gc), ptr(bc), ptr(wm), ptr(v), s, n, np_, stream())
    want_v = (x @ w_m.double().T).view(s, n, 8, 32).permute(2, 0, 3, 1)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    assert rel_l2(v[..., :n].cpu().double(), want_v) < 4e-3
    assert ((v[..., n:] == 7.0) | (v[..., n:] == 0.0)).all()       # padding tokens: zeros, or left alone
    o = torch.randn(8, s, 32, np_, generator=g).bfloat16()
    o[..., n:] = float("nan")                                      # without a say in any token's update
    want = m.double() + (torch.sigmoid(x @ w_g.double().T) * o[..., :n].double().permute(1, 3, 0, 2).reshape(s, n, 256)) @ w_o.double().T
    oc = o.cuda()
    call("b200pf_pwa_output", ptr(mc), ptr(gc), ptr(bc), ptr(wg), ptr(wo), ptr(oc), s, n, np_, stream())
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    assert rel_l2(mc.cpu().double() - m.double(), want - m.double()) < 8e-3


def test_refused_before_launch():
    t = torch.zeros(64, 64, device="cuda")
    for args in (("b200pf_pwa_value", ptr(t), ptr(t), ptr(t), ptr(t), ptr(t), 4, 9, 12), ("b200pf_pwa_output", ptr(t), ptr(t), ptr(t), ptr(t), ptr(t), ptr(t), 4, 9, 8),
                 ("b200pf_msa_transition", ptr(t), ptr(t), None, ptr(t), ptr(t), 4)):
        with pytest.raises(RuntimeError):
            call(*args, stream())
