"""Packing of the fp32-accurate path's weights: bounds and 16-bit parts of a list of tensors against the same in torch, over sizes that
fill a block's share of rows and values and one more, rows in turns of 32, zeros, infinities and NaN, and more items than one launch takes.
Parts and vectors are exact (one rounding each, the same in torch); a row norm is a sum of at most 1536 squares in another order: 1e-4."""
import ctypes as C

import pytest
import torch

from tt_boltz_b200 import _lib

pytestmark = pytest.mark.gpu
SIZES = [(1, 1), (1, 64), (7, 33), (8, 64), (9, 128), (64, 32), (65, 31), (64, 33), (512, 256), (1536, 384), (384, 1536)]


def _stats(wanted):
    items = [_lib.StatItem(w.data_ptr(), None if b is None else b.data_ptr(), w.numel() // w.shape[-1], w.shape[-1]) for w, b in wanted]
    out = torch.empty(len(items), 3, device="cuda")
    _lib.call("b200pf_weight_stats", (_lib.StatItem * len(items))(*items), len(items), out.data_ptr(), _lib.stream())
    return out.cpu()


def test_bounds():
    g = torch.Generator().manual_seed(0)
    wanted = [(torch.randn(r, c, generator=g).cuda() * 10.0 ** (i % 7 - 3), None) for i, (r, c) in enumerate(SIZES * 7)]
    wanted += [(torch.randn(c, generator=g).cuda(), torch.randn(c, generator=g).cuda()) for c in (64, 128, 256, 384)]
    assert len(wanted) > 64
    want = torch.tensor([[float(w.abs().max()), float(w.reshape(-1, w.shape[-1]).norm(dim=1).max()),
                          0.0 if b is None else float((w.numel() ** 0.5 * w.abs() + b.abs()).max())] for w, b in wanted])
    assert torch.allclose(_stats(wanted), want, rtol=1e-4, atol=0)


@pytest.mark.parametrize("odd, top", [(float("inf"), "inf"), (float("-inf"), "inf"), (float("nan"), "nan"), (0.0, "0.0")])
def test_bounds_of_odd_values(odd, top):
    w = torch.zeros(20, 70)
    w[11, 69] = odd
    got = _stats([(w.cuda(), None)])[0]
    assert str(float(got[0])) == str(float(got[1])) == top


def test_parts_and_vectors():
    g = torch.Generator().manual_seed(1)
    src = [torch.randn(r, c, generator=g).cuda() * 10.0 ** (i % 5 - 2) for i, (r, c) in enumerate(SIZES * 6)]
    items, check = [], []
    for i, w in enumerate(src):
        factor, scale = (1.0, 1.4426950408889634)[i % 2], 2.0 ** (i % 9 - 4)
        turns = i % 3 == 0 and w.shape[0] % 32 == 0
        v = (w * torch.tensor(factor, device="cuda")) * scale
        hi = v.half()
        lo = (v - hi.float()).half()
        rows, k = w.shape
        if i % 4 == 1:
            dst = torch.full((rows + 1, k), 5.0, device="cuda")
            items.append(_lib.PackItem(w.data_ptr(), dst.data_ptr(), 0, rows, k, 0, factor, scale, 0, 0))
            items.append(_lib.PackItem(None, dst.data_ptr() + 4 * rows * k, 0, 1, k, 0, 1.0, 1.0, 0, 0))
            check.append((dst, torch.cat([v, torch.zeros(1, k, device="cuda")])))
        else:
            row0, total = (32, 2 * rows) if turns else (3, rows + 3)
            dst = torch.full((2, total, k), 5.0, dtype=torch.float16, device="cuda")
            want = dst.clone()
            at = torch.arange(rows, device="cuda")
            at = row0 + (at // 32 * 64 + at % 32 if turns else at)
            want[0, at], want[1, at] = hi, lo
            items.append(_lib.PackItem(w.data_ptr(), dst.data_ptr(), total * k, rows, k, row0, factor, scale, 2, int(turns)))
            check.append((dst, want))
    assert len(items) > 64
    _lib.call("b200pf_pack_parts", (_lib.PackItem * len(items))(*items), len(items), _lib.stream())
    for i, (got, want) in enumerate(check):
        assert torch.equal(got, want), i


def test_refused_before_launch():
    w = torch.zeros(33, 64, device="cuda")
    bad = [_lib.PackItem(w.data_ptr(), w.data_ptr(), 0, 33, 64, 0, 1.0, 1.0, 2, 1), _lib.PackItem(w.data_ptr(), None, 0, 1, 64, 0, 1.0, 1.0, 0, 0)]
    for item in bad:
        with pytest.raises(RuntimeError):
            _lib.call("b200pf_pack_parts", C.byref(item), 1, _lib.stream())
    with pytest.raises(RuntimeError):
        _lib.call("b200pf_weight_stats", C.byref(_lib.StatItem(w.data_ptr(), w.data_ptr(), 33, 64)), 1, w.data_ptr(), _lib.stream())
