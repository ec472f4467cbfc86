"""The MSA embedding in one kernel against one-hot, concatenation and linear in 64 bits, with and without the paired feature: one row, rows
that do not fill a block, more than a lane takes at once.  The projected single representation comes from the linear kernel as it does in the
module; on top of it are four rounded additions, each half an ulp of at most the sum of the terms' sizes: 2^-22 of that.  A residue outside the classes makes its
row NaN and is reported, and a call of the module with one raises; features of another shape or type are refused."""
import threading

import pytest
import torch

from tt_boltz_b200 import B200MSAModule, _lib, ops
from tt_boltz_b200._lib import call, ptr, stream

pytestmark = pytest.mark.gpu


def case(s, n, paired):
    g = torch.Generator().manual_seed(100 * s + n)
    mod = B200MSAModule(64, 128, 384, 1, use_paired_feature=paired)
    with torch.no_grad():
        for p in (mod.s_proj.weight, mod.msa_proj.weight):
            p.copy_(torch.randn(p.shape, generator=g) * 0.1)
    feats = {"msa": torch.randint(0, 33, (1, s, n), generator=g), "has_deletion": (torch.rand(1, s, n, generator=g) < 0.2),
             "deletion_value": torch.rand(1, s, n, generator=g).double(), "msa_paired": torch.randint(0, 2, (1, s, n), generator=g)}
    return mod.cuda(), torch.randn(1, n, 384, generator=g).cuda(), {k: v.cuda() for k, v in feats.items()}


@pytest.mark.parametrize("paired", [True, False])
@pytest.mark.parametrize("s, n", [(1, 1), (3, 5), (1, 17), (7, 64), (33, 130), (600, 301)])
def test_embedding(s, n, paired):
    mod, emb, feats = case(s, n, paired)
    raw = [torch.nn.functional.one_hot(feats["msa"][0], 33).double()] + [feats[k][0][..., None].float().double() for k in ("has_deletion", "deletion_value")]
    raw += [feats["msa_paired"][0][..., None].double()] if paired else []
    w = mod.msa_proj.weight.detach().double()
    e = ops.f32_linear(emb[0], mod.s_proj.weight.detach()).double()[None]
    raw = torch.cat(raw, -1)
    got = mod.embed(emb, feats)
    assert _lib.device_status() == 0
    assert bool(((got.double() - (raw @ w.t() + e)).abs() <= 2.0 ** -22 * (raw.abs() @ w.abs().t() + e.abs())).all())


def test_what_is_refused():
    mod, emb, feats = case(4, 9, True)
    with torch.no_grad():
        good = mod.embed(emb, feats)
        feats["msa"][0, 2, 3] = 33
        got = mod.embed(emb, feats)
        assert _lib.device_status() == 2
        same = torch.ones(4, 9, dtype=torch.bool)
        same[2, 3] = False
        assert torch.equal(got[same], good[same])
        for key, value in (("msa", feats["msa"].int()), ("msa_paired", feats["msa_paired"][:, :3]), ("deletion_value", feats["deletion_value"][:, :, :5])):
            with pytest.raises(RuntimeError):
                mod.embed(emb, {**feats, key: value})
        with pytest.raises(RuntimeError):
            mod.embed(emb[:, :5], feats)
    assert _lib.device_status() == 0


def module_case(residue):
    mod, emb, feats = case(5, 9, True)
    with torch.no_grad():
        for p in mod.layers.parameters():
            p.normal_(0.0, 0.05) if p.dim() == 2 else p.fill_(1.0)
    feats.update({"msa_mask": torch.ones(1, 5, 9, device="cuda"), "token_pad_mask": torch.ones(1, 9, device="cuda")})
    bad = {**feats, "msa": feats["msa"].clone()}
    bad["msa"][0, 4, 8] = residue
    return mod, (torch.randn(1, 9, 9, 128, device="cuda"), emb), feats, bad


@pytest.mark.parametrize("residue", [-1, 33, 1 << 40])
def test_a_call_with_a_bad_residue_raises(residue):
    mod, args, feats, bad = module_case(residue)
    good = mod(*args, feats)
    with pytest.raises(RuntimeError, match="residues"):
        mod(*args, bad)
    assert torch.equal(mod(*args, feats), good)                      # nothing is left behind
    assert bool(torch.isfinite(good).all()) and _lib.device_status() == 0


def test_a_captured_call_with_a_bad_residue_is_no_number():
    mod, args, feats, bad = module_case(33)
    mod(*args, feats)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        z = mod(*args, bad)
    graph.replay()
    assert _lib.device_status() == 2
    assert bool(torch.isnan(z).all())


@pytest.mark.parametrize("s, n", [(1, 1), (3, 5), (33, 130), (600, 301)])
def test_token_rows(s, n):
    """One rounded addition a value: torch's."""
    torch.manual_seed(n)
    m, e = torch.randn(s + 1, n, 64, device="cuda"), torch.randn(n, 64, device="cuda")
    want = torch.cat([m[:s] + e, m[s:]])
    call("b200pf_msa_add_token_rows", ptr(m), ptr(e), s, n, stream())
    assert torch.equal(m, want)


def test_a_call_beside_another_threads_capture():
    """The wait for the embedding's answer is no obstacle to a capture that another thread has under way, nor that to it."""
    mod, args, feats, _ = module_case(0)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        want = [mod(*args, feats) for _ in range(3)][-1]
    torch.cuda.synchronize()
    got, x = [], torch.ones(8, device="cuda")

    def work():
        try:
            with torch.cuda.stream(side):
                got.append(mod(*args, feats))
        except RuntimeError as e:
            got.append(e)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="global"):
        y = x + 1
        thread = threading.Thread(target=work)
        thread.start()
        thread.join()
    graph.replay()
    torch.cuda.synchronize()
    assert isinstance(got[0], torch.Tensor), got[0]
    assert torch.equal(got[0], want) and bool((y == 2).all())
