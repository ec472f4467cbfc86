"""Workspaces of the fp32-accurate path: one for more rows serves fewer, and a transition refuses one that is too small before any
CUDA call.  On the GPU, a transition at the row counts around the limit of its partial sums stays inside what it asked for."""
import ctypes as C

import pytest
import torch

from tt_boltz_b200 import _lib, ops, weights


@pytest.mark.parametrize("c, hidden", [(64, 256), (128, 512), (256, 1024), (384, 1536)])
def test_workspaces_grow_with_their_rows(c, hidden):
    lib = _lib.load()
    for size in (lambda r: lib.b200pf_split_transition_workspace(r, c, hidden), lambda r: lib.b200pf_single_track_workspace(r, c, hidden),
                 lambda r: lib.b200pf_single_track_rows_workspace(r, c, hidden), lambda r: lib.b200pf_split_pair_workspace(r, c, 0, 0, hidden)):
        sizes = [size(r) for r in range(1, 2200)]
        assert all(a <= b for a, b in zip(sizes, sizes[1:]))


@pytest.mark.parametrize("rows", [1, 2026, 2048, 2049, 1 << 20])
def test_a_short_workspace_is_refused(rows):
    lib = _lib.load()
    w = _lib.SplitTransitionWeights(c=128, hidden=512)
    buf = (C.c_char * 64)()
    p = (C.addressof(buf) + 15) // 16 * 16                      # never dereferenced
    short = lib.b200pf_split_transition_workspace(rows, 128, 512) - 1
    assert lib.b200pf_split_transition(p, rows, C.byref(w), p, short, None) != 0
    assert "too few" in _lib.last_error()


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [2025, 2026, 2048, 2049])
def test_transition_stays_inside_its_workspace(rows):
    from oracle import pairformer_oracle as orc
    from tests.test_gpu_split import TOL, layer, rel_l2
    dev, guard = torch.device("cuda:0"), 1 << 20
    sd = layer(128, 4)
    x = torch.randn(rows, 128, generator=torch.Generator().manual_seed(rows)).to(dev)
    pack = weights.pack_split_transition(sd, "transition_z.", dev)
    nbytes = _lib.load().b200pf_split_transition_workspace(rows, 128, 512)
    ws = torch.full((nbytes + guard,), 0xA5, dtype=torch.uint8, device=dev)
    out = x.clone()
    _lib.call("b200pf_split_transition", _lib.ptr(out), rows, C.byref(pack.struct), _lib.ptr(ws), nbytes, _lib.stream())
    assert bool((ws[nbytes:] == 0xA5).all())
    same = x.clone()
    ops.transition_split(same, pack, ops.Scratch(dev))
    assert torch.equal(same, out)
    want = orc.transition(x.double(), {k: v.double().to(dev) for k, v in sd.items()}, "transition_z")
    slack = float(2.0 ** -24 * x.double().norm() / want.norm())
    assert rel_l2(out.double() - x.double(), want) < TOL + slack
    assert _lib.device_status() == 0
