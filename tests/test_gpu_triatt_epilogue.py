"""The triangle-attention epilogue at the edges of its rules: 32, 64 or 128 rows a tile by how many fill the multiprocessors, rows short of a
tile, one tile per CTA and several; into the residual and as an update of its own.  o * g is one fp32 product rounded to bf16; 128 exact
products per value, summed in fp32 by truncating MMAs of 16: at most 8 + 16 ulps of the sum of their magnitudes, 2^-18 of it, then half an ulp
of the residual, or half an ulp of bf16's 8 bits of the update, at most 2^-8 of it."""
import pytest
import torch

from tt_boltz_b200 import _lib
from tt_boltz_b200._lib import call, ptr, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("update", [False, True])
@pytest.mark.parametrize("per_sm, rest", [(0, 1), (0, 31), (0, 32), (0, 33), (32, 0), (32, 1), (64, 0), (64, 1), (128, -5), (128, 1), (700, 37)])
def test_epilogue(per_sm, rest, update):
    dev = torch.device("cuda:0")
    rows = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + rest
    g = torch.Generator(device=dev).manual_seed(rows)
    rand = lambda *s: torch.randn(*s, device=dev, generator=g)
    o, gate, w = rand(rows, 128).bfloat16(), torch.sigmoid(rand(rows, 128)).bfloat16(), (rand(128, 128) * 0.1).bfloat16()
    og = (o.float() * gate.float()).bfloat16().double()
    want, size = og @ w.double().t(), og.abs() @ w.double().abs().t()
    if update:
        out = torch.full((rows + 1, 128), 7.0, device=dev, dtype=torch.bfloat16)
        call("b200pf_triatt_epilogue_update", ptr(out), ptr(o), ptr(gate), ptr(w), rows, stream())
        bound = 2.0 ** -18 * size + 2.0 ** -8 * want.abs()
    else:
        out = rand(rows + 1, 128)
        out[rows] = 7.0
        want = want + out[:rows].double()
        call("b200pf_triatt_epilogue", ptr(out), ptr(o), ptr(gate), ptr(w), rows, stream())
        bound = 2.0 ** -18 * size + 2.0 ** -24 * want.abs()
    assert _lib.device_status() == 0
    assert bool(((out[:rows].double() - want).abs() <= bound).all())
    assert bool((out[rows] == 7.0).all())                       # nothing behind the last row
