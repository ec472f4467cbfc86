"""The MSA embedding's features come from one device: its kernel takes their addresses, and another device's memory behind one is a fault and
not an error message.  (Without a GPU: the check stands before any kernel.)"""
import pytest
import torch

from tt_boltz_b200 import B200MSAModule


@pytest.mark.parametrize("elsewhere", ["has_deletion", "deletion_value", "msa_paired", "emb"])
def test_features_of_another_device_are_refused(elsewhere):
    mod = B200MSAModule(64, 128, 384, 1)
    feats = {"msa": torch.zeros(1, 3, 5, dtype=torch.int64), **{k: torch.zeros(1, 3, 5) for k in ("has_deletion", "deletion_value", "msa_paired")}}
    emb = torch.zeros(1, 5, 384, device="meta" if elsewhere == "emb" else "cpu")
    if elsewhere != "emb":
        feats[elsewhere] = feats[elsewhere].to("meta")
    with pytest.raises(RuntimeError, match="are on cpu"):
        mod.embed(emb, feats)
