"""Triangle attention of the fp32-accurate path where scores grow past the point at which a reference with the parts' shift of 14 rounds:
the probabilities' fp16 parts must not overflow, whatever the scores' size.  With the LayerNorm gain times g the scores grow with g * g."""
import pytest
import torch

from tests.test_gpu_split import inputs, layer
from tt_boltz_b200 import _lib, ops, weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gain", [1e2, 3e3, 5e3, 1e4, 2e4, 5e4])
def test_large_scores_stay_finite(gain):
    dev, n = torch.device("cuda:0"), 130
    sd = layer(64, 4)
    sd["tri_att_start.layer_norm.weight"] = sd["tri_att_start.layer_norm.weight"] * gain
    _, z, pm, _ = inputs(n, 64)
    out = z.to(dev)
    ops.tri_att_split(out, pm.to(torch.uint8).to(dev), weights.pack_split_triatt(sd, "tri_att_start.", dev), False, ops.Scratch(dev))
    assert bool(torch.isfinite(out).all())
    assert _lib.device_status() == 0
