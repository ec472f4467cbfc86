"""One call per block against the sub-operations one by one (the same kernels: bit-identical), and the single track beside the pair
track against behind it (the same kernels on another stream: bit-identical)."""
import pytest
import torch

from tt_boltz_b200 import B200PairformerModule, _lib, ops, pairformer, synthetic

pytestmark = pytest.mark.gpu


def _module(blocks, precision="bf16"):
    mod = B200PairformerModule(384, 128, blocks, v2=True, precision=precision)
    mod.load_state_dict(synthetic.make_weights(blocks, seed=3, std=0.05, affine_jitter=0.2), strict=True)
    return mod


def _inputs(n):
    s, z = synthetic.make_inputs(n, seed=n)
    m, pm = synthetic.tail_padding_mask(n, n // 8)
    return [t.cuda() for t in (s, z, m, pm)]


@pytest.mark.parametrize("n", [1, 17, 130])
def test_block_call_is_the_sub_operations(n):
    mod = _module(2)
    args = _inputs(n)
    one = mod(*args)
    _lib.timer = _lib.KernelTimer()          # with a timer every sub-operation is a call of its own
    try:
        many = mod(*args)
        assert "b200pf_trimul_producer" in _lib.timer.summary()
    finally:
        _lib.timer = None
    assert _lib.device_status() == 0
    assert torch.equal(one[0], many[0]) and torch.equal(one[1], many[1])


@pytest.mark.parametrize("n", [5, 64, 128, 129])
@pytest.mark.parametrize("precision", ["bf16", "mxfp8"])
def test_single_track_beside_the_pair_track(n, precision, monkeypatch):
    mod = _module(5, precision)              # odd: both bias buffers are taken, one of them three times
    args = _inputs(n)
    monkeypatch.setenv("B200PF_SIDE_TRACK", "0")
    behind = mod(*args)
    monkeypatch.setenv("B200PF_SIDE_TRACK", "1")
    for _ in range(3):
        beside = mod(*args)
        assert torch.equal(behind[0], beside[0]) and torch.equal(behind[1], beside[1])
    monkeypatch.delenv("B200PF_SIDE_TRACK")
    auto = mod(*args)
    assert torch.equal(behind[0], auto[0]) and torch.equal(behind[1], auto[1])
    assert pairformer._side_track_wanted(n) and not pairformer._side_track_wanted(1 + pairformer.SIDE_TRACK_TOKENS)
    assert _lib.device_status() == 0


@pytest.mark.parametrize("n", [100, 128])
def test_single_track_beside_a_wide_pair_track(n, monkeypatch):
    """256 pair channels: the single track's kernels take the whole chip there, next to 128 channels they keep to a part of it."""
    mod = B200PairformerModule(384, 256, 3, pairwise_num_heads=8, v2=True, precision="auto")
    mod.load_state_dict(synthetic.make_weights(3, seed=3, std=0.05, affine_jitter=0.2, c_z=256, tri_heads=8), strict=True)
    s, z = synthetic.make_inputs(n, c_z=256, seed=n)
    args = [t.cuda() for t in (s, z, *synthetic.tail_padding_mask(n, n // 8))]
    monkeypatch.setenv("B200PF_SIDE_TRACK", "0")
    behind = mod(*args)
    monkeypatch.setenv("B200PF_SIDE_TRACK", "1")
    beside = mod(*args)
    assert torch.equal(behind[0], beside[0]) and torch.equal(behind[1], beside[1])
    assert _lib.device_status() == 0


def test_a_failing_layer_leaves_nothing_running_beside(monkeypatch):
    mod = _module(3)
    args = _inputs(40)
    want = mod(*args)
    calls = []

    def broken(self, *a):
        calls.append(1)
        if len(calls) == 2:
            raise RuntimeError("no")
        return real(self, *a)
    real = ops.PairBlock.run
    monkeypatch.setattr(ops.PairBlock, "run", broken)
    with pytest.raises(RuntimeError, match="no"):
        mod(*args)
    monkeypatch.undo()
    got = mod(*args)
    assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])


def test_a_timer_sees_the_single_track():
    """Its kernels run behind the pair track then, as entry points of their own: an event pair on the pair stream would miss them on another."""
    mod = _module(3)
    args = _inputs(40)
    want = mod(*args)
    _lib.timer = _lib.KernelTimer()
    try:
        got = mod(*args)
        seen = _lib.timer.summary()
    finally:
        _lib.timer = None
    assert seen["b200pf_single_track_rows"][1] == 3 and "b200pf_single_track_beside" not in seen
    assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])
