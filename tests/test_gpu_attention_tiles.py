"""The attention core where its one-pass softmax takes its references and exclusions: a line's first 64-key tile (reference from
its first 32 keys), the ragged last tile, and tiles given back to the two-pass path because their reference is a masked key's
score.  Against the fp32 tier on the same z; the bf16 tier's tolerance for one sub-operation's update (2e-2: q, k, v, the
probabilities and the output are bf16; measured 4e-3).  Scores stay of order one: a score s carries the rounding 2^-9 |s| of q and
k, so with scores of hundreds the comparison would be of that rounding and not of the tiles."""
import pytest
import torch

from tests.conftest import rel_l2
from tt_boltz_b200 import _lib, ops, synthetic, weights

pytestmark = pytest.mark.gpu


def _mask(kind, n):
    m = torch.ones(n, n, dtype=torch.uint8)
    if kind == "late":              # nothing to attend to before the last key
        m[:, : n - 1] = 0
    elif kind == "second_half":     # the first tile's reference comes from masked keys only
        m[:, : min(32, n - 1)] = 0
    elif kind == "none":
        m[:, :] = 0
    elif kind == "block":           # two groups that see only their own (a general mask: tiles fully masked for some lines)
        h = n // 2
        m[:h, h:] = 0
        m[h:, :h] = 0
    return m


@pytest.mark.parametrize("n, kind", [(1, "ones"), (31, "ones"), (33, "second_half"), (63, "late"), (64, "second_half"), (65, "ones"), (95, "late"),
                                     (96, "block"), (97, "second_half"), (129, "block"), (161, "none"), (193, "late"), (203, "ones")])
def test_first_and_ragged_tiles(n, kind):
    dev = torch.device("cuda")
    sd = synthetic.make_weights(1, seed=7, std=0.05, affine_jitter=0.2)
    sd = {k[len("layers.0."):]: v for k, v in sd.items()}
    _, z = synthetic.make_inputs(n, seed=n, with_s=False)
    mask = _mask(kind, n).to(dev)
    masks, ws = ops.PairMasks(mask), ops.Workspace(n, dev)
    for pre, ending in (("tri_att_start.", False), ("tri_att_end.", True)):
        zd, zf = z[0].to(dev).clone(), z[0].to(dev).clone()
        ops.tri_att_bf16(zd, masks, weights.pack_triatt(sd, pre, dev), ws, ending)
        ops.tri_att_f32(zf, mask, weights.to_device_f32(sd, pre, dev), ending)
        torch.cuda.synchronize()
        assert _lib.device_status() == 0
        upd, want = (zd.cpu() - z[0]), (zf.cpu() - z[0])
        assert torch.isfinite(upd).all()
        assert rel_l2(upd, want) < 2e-2


@pytest.mark.parametrize("n, kind", [(64, "ones"), (128, "late"), (128, "block"), (192, "none"), (192, "second_half"), (256, "ones")])
def test_lines_of_whole_tiles(n, kind):
    """The form of the core for token counts that are multiples of 64, which has no test for a short last tile."""
    test_first_and_ragged_tiles(n, kind)
