"""The MSA transition and the averaging's output with gates far out on both sides, among them some beyond where the exponential stops growing,
next to ones around zero.  Gate inputs of standard deviation 20, rounded to 1.6e-3 of that by their bf16
factors (two in quadrature over 64 channels): silu's slope is at most 1.1 and its root mean square 0.7 of the input's, 2.5e-3; the sigmoid's
slope is 0.25 for the sixth of the inputs below 4 and its root mean square 0.7, 4.6e-3; with the other factors' and the roundings behind, 8e-3
covers both."""
import pytest
import torch
import torch.nn.functional as F

from tests.conftest import rel_l2
from tt_boltz_b200 import _lib
from tt_boltz_b200._lib import call, ptr, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s, n", [(1, 5), (7, 130)])
def test_wide_gates(s, n):
    g = torch.Generator().manual_seed(n)
    m, gam, bet = torch.randn(s, n, 64, generator=g), torch.ones(64), torch.zeros(64)
    w = lambda rows, cols, std: (torch.randn(rows, cols, generator=g) * std).bfloat16()
    fc1, fc2, fc3 = w(256, 64, 2.5), w(256, 64, 0.15), w(64, 256, 0.15)
    x = F.layer_norm(m.double(), (64,), gam.double(), bet.double(), 1e-5)
    gate = x @ fc1.double().T
    assert gate.min() < -43 and gate.max() > 43
    gc, bc, w1, w3 = gam.cuda(), bet.cuda(), fc1.cuda(), fc3.cuda()
    w12 = torch.stack([fc1.view(4, 64, 64), fc2.view(4, 64, 64)], 1).contiguous().cuda()
    mt = m.cuda()
    call("b200pf_msa_transition", ptr(mt), ptr(gc), ptr(bc), ptr(w12), ptr(w3), s * n, stream())
    np_ = (n + 7) // 8 * 8
    o = torch.randn(8, s, 32, np_, generator=g).bfloat16()
    oc, mo = o.cuda(), m.cuda()
    call("b200pf_pwa_output", ptr(mo), ptr(gc), ptr(bc), ptr(w1), ptr(w3), ptr(oc), s, n, np_, stream())
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    assert rel_l2(mt.cpu().double() - m.double(), (F.silu(gate) * (x @ fc2.double().T)) @ fc3.double().T) < 8e-3
    avg = o[..., :n].double().permute(1, 3, 0, 2).reshape(s, n, 256)
    assert rel_l2(mo.cpu().double() - m.double(), (torch.sigmoid(gate) * avg) @ fc3.double().T) < 8e-3


def test_tokens_are_independent():
    """What the output kernel adds to a token hangs on that token alone: the same bits whatever stands at its neighbours, a NaN included."""
    s, n, np_ = 40, 303, 304
    g = torch.Generator().manual_seed(1)
    m, other = torch.randn(s, n, 64, generator=g).cuda(), torch.randn(s, n, 64, generator=g).cuda()
    gam, bet, o = torch.ones(64).cuda(), torch.zeros(64).cuda(), torch.randn(8, s, 32, np_, generator=g).bfloat16().cuda()
    wg, wo = (torch.randn(256, 64, generator=g) * 0.3).bfloat16().cuda(), (torch.randn(64, 256, generator=g) * 0.1).bfloat16().cuda()

    def output(x):
        x = x.clone()
        call("b200pf_pwa_output", ptr(x), ptr(gam), ptr(bet), ptr(wg), ptr(wo), ptr(o), s, n, np_, stream())
        return x
    want = output(m)
    for first in (0, 1):
        x = m.clone()
        x[:, first::2] = other[:, first::2]
        assert torch.equal(output(x)[:, 1 - first::2], want[:, 1 - first::2])
        x[:, first::2] = float("nan")
        got = output(x)
        assert torch.equal(got[:, 1 - first::2], want[:, 1 - first::2]) and bool(torch.isnan(got[:, first::2]).all())
    assert _lib.device_status() == 0


def test_far_gates_go_on_falling():
    """silu at some -50, times a value of some 1e18: -50 e^-50, to the tenth of an argument that its bf16 factors leave open and a third more."""
    g = torch.Generator().manual_seed(2)
    m, gam, bet = torch.randn(3, 64, generator=g), torch.ones(64), torch.zeros(64)
    x = F.layer_norm(m.double(), (64,), gam.double(), bet.double(), 1e-5)
    fc1, fc2, fc3 = torch.zeros(256, 64), torch.zeros(256, 64), torch.zeros(64, 256)
    v = x[0].float() / 64                                            # x is LayerNorm's: v . x is 1 for row 0
    fc1[0], fc2[0], fc3[0, 0] = -50 * v, 1e18 * v, 1.0
    fc1, fc2, fc3 = fc1.bfloat16(), fc2.bfloat16(), fc3.bfloat16()
    w12 = torch.stack([fc1.view(4, 64, 64), fc2.view(4, 64, 64)], 1).contiguous().cuda()
    mt, gc, bc, w3 = m.cuda(), gam.cuda(), bet.cuda(), fc3.cuda()
    call("b200pf_msa_transition", ptr(mt), ptr(gc), ptr(bc), ptr(w12), ptr(w3), 3, stream())
    gate, value = x[0] @ fc1[0].double(), x[0] @ fc2[0].double()
    want = float(gate * torch.exp(gate) * value)
    got = float(mt[0, 0].cpu().double() - m[0, 0].double())
    assert -0.1 < want < -1e-3 and abs(got / want - 1) < 0.4, (got, want)
    assert _lib.device_status() == 0
