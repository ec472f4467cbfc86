"""Timed cases of the Pairformer path: what a structure-prediction program has this package do, by call site.

Every case is one call of a public module on inputs that are already on the GPU.  The kinds are the places in a
Boltz-2 fold (and in the sibling models that share the blocks) that call the package:

* ``pairformer``  the trunk (64 blocks) and the confidence head (8 blocks): single and pair track, bf16 tier
* ``affinity``    the pair-only stack of the affinity head, with a mask that keeps protein-ligand pairs only
* ``fast``        a slice of the trunk for large complexes with MXFP8 triangle multiplications
* ``recycle``     the trunk inside its recycling loop, and the distogram read off the resident pair tensor
* ``template``    the pair-only stack of the template module (pair width 64, fp32 kernels)
* ``wide``        blocks of a sibling trunk with pair width 256 and 8 triangle heads (fp32 kernels)
* ``fold``        attention-free blocks of a folding trunk with pair width 256 (fp32 kernels)
* ``msa``         the MSA module: 4 blocks on embedded features

Sizes run from a peptide (some 30 tokens) to a large complex (2048); most proteins lie between 100 and 600 tokens,
and hardly any token count is a multiple of anything.  Weights are drawn per parameter as the benchmark draws them
(matrices N(0, 0.02), 0.05 in the MSA module), with gains around 1 and offsets around 0.
"""
from __future__ import annotations

import math

import torch

from tt_boltz_b200 import (B200DistogramModule, B200MSAModule, B200PairformerModule, B200PairformerNoSeqModule,
                           B200PairUpdateBlock, B200RecyclingTrunk)

C_S, C_Z, C_M = 384, 128, 64


def listed():
    return [
        # confidence head on a short peptide: the smallest call, bound by launches
        {"name": "confidence_n45", "kind": "pairformer", "n": 45, "blocks": 8, "pad": 0},
        # affinity head on the crop around a ligand
        {"name": "affinity_n117", "kind": "affinity", "n": 117, "blocks": 8, "ligand": 29},
        # trunk of an ordinary protein, a token count with no factor of two
        {"name": "trunk_n203", "kind": "pairformer", "n": 203, "blocks": 64, "pad": 0},
        # trunk of a mid-sized complex, padded as a batching data loader leaves it
        {"name": "trunk_n400", "kind": "pairformer", "n": 400, "blocks": 64, "pad": 16},
        # the headline configuration: the whole trunk at 1024 tokens
        {"name": "trunk_n1024", "kind": "pairformer", "n": 1024, "blocks": 64, "pad": 0},
        # large complex in the fast tier, 5 % of its tokens masked at random; 4 of the trunk's 48 blocks
        {"name": "fast_n2048", "kind": "fast", "n": 2048, "blocks": 4, "drop": 0.05},
        # two passes of the recycling loop and the distogram, on a two-chain complex
        {"name": "recycle_n509", "kind": "recycle", "n": 509, "blocks": 16, "recycles": 1},
        # template module, once per recycle and template
        {"name": "template_n292", "kind": "template", "n": 292, "blocks": 2, "pad": 0},
        # sibling trunk with a 256-wide pair tensor, 2 of its 48 blocks
        {"name": "wide_n256", "kind": "wide", "n": 256, "blocks": 2, "pad": 8},
        # folding trunk without attention, 4 of its 48 blocks
        {"name": "fold_n331", "kind": "fold", "n": 331, "blocks": 4, "pad": 0},
        # MSA module on a shallow alignment
        {"name": "msa_s122_n171", "kind": "msa", "s": 122, "n": 171, "blocks": 4, "pad": 0},
        # MSA module at the default subsampling depth
        {"name": "msa_s1024_n600", "kind": "msa", "s": 1024, "n": 600, "blocks": 4, "pad": 24},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pairformer", "pairformer", "pairformer", "affinity", "fast", "recycle", "template", "wide", "fold", "msa", "msa"])
    if kind == "pairformer":
        n = _log_int(rng, 30, 1024)
        return {"kind": kind, "n": n, "blocks": rng.choice([8, 64]), "pad": rng.choice([0, 0, rng.randrange(1, 1 + n // 8)])}
    if kind == "affinity":
        n = _log_int(rng, 40, 512)
        return {"kind": kind, "n": n, "blocks": rng.choice([4, 8]), "ligand": rng.randrange(4, 1 + n // 3)}
    if kind == "fast":
        return {"kind": kind, "n": _log_int(rng, 256, 2048), "blocks": rng.randrange(2, 5), "drop": rng.choice([0.0, 0.05])}
    if kind == "recycle":
        return {"kind": kind, "n": _log_int(rng, 40, 640), "blocks": 16, "recycles": rng.randrange(0, 4)}
    if kind == "template":
        n = _log_int(rng, 48, 640)
        return {"kind": kind, "n": n, "blocks": 2, "pad": rng.choice([0, rng.randrange(1, 1 + n // 8)])}
    if kind == "wide":
        n = _log_int(rng, 40, 320)
        return {"kind": kind, "n": n, "blocks": 2, "pad": rng.choice([0, rng.randrange(1, 1 + n // 8)])}
    if kind == "fold":
        n = _log_int(rng, 40, 400)
        return {"kind": kind, "n": n, "blocks": 4, "pad": rng.choice([0, rng.randrange(1, 1 + n // 8)])}
    n = _log_int(rng, 40, 768)
    return {"kind": kind, "s": _log_int(rng, 8, min(4096, 1048576 // n)), "n": n, "blocks": 4, "pad": rng.choice([0, rng.randrange(1, 1 + n // 8)])}


# ------------------------------------------------------------------------------------------------
# what a program holds before the call
# ------------------------------------------------------------------------------------------------
def _fill(module: torch.nn.Module, gen: torch.Generator, std: float) -> torch.nn.Module:
    """Random weights in place of the freshly built module's, as a checkpoint would put them there."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            p.requires_grad_(False)
            p.normal_(0.0, std if p.dim() == 2 else 0.1, generator=gen)
            if p.dim() == 1 and name.endswith("weight"):
                p += 1.0
    return module.eval()


def _module(case):
    kind, blocks = case["kind"], case["blocks"]
    if kind == "pairformer":
        return B200PairformerModule(C_S, C_Z, blocks, v2=True, precision="bf16")
    if kind == "affinity":
        return B200PairformerNoSeqModule(C_Z, blocks, precision="bf16")
    if kind == "fast":
        return B200PairformerModule(C_S, C_Z, blocks, v2=True, precision="mxfp8")
    if kind == "recycle":
        return torch.nn.ModuleDict({"trunk": B200RecyclingTrunk(B200PairformerModule(C_S, C_Z, blocks, v2=True, precision="bf16")),
                                    "distogram": B200DistogramModule(C_Z, 64, 1)})
    if kind == "template":
        return B200PairformerNoSeqModule(64, blocks, precision="auto")
    if kind == "wide":
        return B200PairformerModule(C_S, 256, blocks, pairwise_num_heads=8, v2=True, precision="auto")
    if kind == "fold":
        return torch.nn.ModuleList(B200PairUpdateBlock(256) for _ in range(blocks))
    return B200MSAModule(C_M, C_Z, C_S, blocks, precision="bf16")


def _width(case) -> int:
    return {"template": 64, "wide": 256, "fold": 256}.get(case["kind"], C_Z)


def _inputs(case, gen, dev):
    """The call's arguments: seeded N(0, 1) tensors and the masks of the kind."""
    kind, n = case["kind"], case["n"]
    rand = lambda *shape: torch.randn(*shape, device=dev, generator=gen)
    out = {"z": rand(1, n, n, _width(case))}
    tok = torch.ones(1, n, device=dev)
    if case.get("pad"):
        tok[:, n - case["pad"]:] = 0
    if case.get("drop"):
        tok = (torch.rand(1, n, device=dev, generator=gen) >= case["drop"]).float()
    out["mask"], out["pair_mask"] = tok, tok[:, :, None] * tok[:, None, :]
    if kind == "affinity":              # pairs between the ligand (the last tokens) and the protein, and within the ligand
        lig = (torch.arange(n, device=dev) >= n - case["ligand"]).float()
        out["pair_mask"] = (lig[None, :, None] + lig[None, None, :] > 0).float()
    if kind in ("pairformer", "fast", "recycle", "wide"):
        out["s"] = rand(1, n, C_S)
    if kind == "msa":
        s = case["s"]
        msa_mask = (torch.rand(1, s, n, device=dev, generator=gen) >= 0.1).float()
        msa_mask[:, 0] = 1.0
        out["emb"] = rand(1, n, C_S)
        out["feats"] = {"msa": torch.randint(0, 33, (1, s, n), device=dev, generator=gen),
                        "has_deletion": (torch.rand(1, s, n, device=dev, generator=gen) < 0.1).float(),
                        "deletion_value": torch.rand(1, s, n, device=dev, generator=gen),
                        "msa_paired": (torch.rand(1, s, n, device=dev, generator=gen) < 0.5).float(),
                        "msa_mask": msa_mask, "token_pad_mask": tok}
    return out


def prepare(case, seed):
    """The module with its weights, warmed up on a small input as a serving program does after loading a checkpoint,
    and the inputs of one call."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    with dev:
        module = _module(case)
    state = {"kind": case["kind"], "recycles": case.get("recycles", 0), "module": _fill(module, gen, 0.05 if case["kind"] == "msa" else 0.02)}
    small = {k: v for k, v in case.items() if k not in ("pad", "drop")}
    small.update({"n": 16, "s": 8, "ligand": 4})
    run({**state, **_inputs(small, gen, dev)})
    state.update(_inputs(case, gen, dev))
    return state


def run(state):
    kind, module, z = state["kind"], state["module"], state["z"]
    if kind in ("pairformer", "fast", "wide"):
        return module(state["s"], z, state["mask"], state["pair_mask"])
    if kind in ("affinity", "template"):
        return module(z, state["pair_mask"])
    if kind == "recycle":
        s, z = module["trunk"](state["s"], z, state["mask"], state["pair_mask"], recycling_steps=state["recycles"])
        return {"s": s, "z": z, "distogram": module["distogram"](z)}
    if kind == "fold":
        for block in module:
            z = block(z, state["pair_mask"])
        return z
    return module(z, state["emb"], state["feats"])


# ------------------------------------------------------------------------------------------------
# work and tolerance
# ------------------------------------------------------------------------------------------------
def _pair_flops(n: int, c: int, attention: bool = True) -> float:
    """Two triangle multiplications, two triangle attentions, the transition (hidden 4 c) on an n x n x c tensor."""
    tri_mul = 2 * n ** 3 * c + 12 * n * n * c * c
    tri_att = 4 * n ** 3 * c + 10 * n * n * c * c + 2 * n * n * c * (c // 32)
    return 2 * tri_mul + (2 * tri_att if attention else 0) + 24 * n * n * c * c


def _single_flops(n: int, c: int) -> float:
    return 10 * n * C_S ** 2 + 4 * n * n * C_S + 32 * n * n * c + 24 * n * C_S ** 2


def _pair_weights(c: int, attention: bool = True) -> int:
    return (12 + (10 if attention else 0) + 12) * c * c


def work(case):
    kind, n, blocks, c = case["kind"], case["n"], case["blocks"], _width(case)
    fused = c == C_Z
    z_bytes = 4 * n * n * c
    single = kind in ("pairformer", "fast", "recycle", "wide")
    flops = blocks * (_pair_flops(n, c, kind != "fold") + (_single_flops(n, c) if single else 0))
    weights = blocks * (_pair_weights(c, kind != "fold") * (2 if fused else 4) + (17 * C_S ** 2 * 4 if single else 0))
    moved = 2 * z_bytes + 4 * n * n + (8 * n * C_S + 4 * n if single else 0)
    if kind == "recycle":
        passes = case["recycles"] + 1
        flops = passes * (flops + 2 * n * n * c * c + 2 * n * C_S ** 2) + 2 * n * n * c * 64
        moved += 4 * n * n * 64
    if kind == "msa":
        s = case["s"]
        rows = s * n
        pwa = rows * (2 * C_M * 512 + 2 * 256 * C_M) + 2 * s * n * n * 256 + 2 * n * n * c * 8
        transition = 6 * rows * C_M * 256
        outer = 2 * rows * C_M * 64 + 2 * s * (32 * n) ** 2 + 2 * n * n * 1024 * c
        flops += blocks * (pwa + transition + outer) + 2 * rows * 36 * C_M
        weights += blocks * 2 * (C_M * 512 + 256 * C_M + 3 * C_M * 256 + 64 * C_M + 1024 * c)
        moved += rows * (8 + 4 * 4) + 4 * n * C_S       # int64 residues and four fp32 features
    return {"bytes": float(moved + weights), "flops": float(flops)}


def tolerance(case):
    """About four times what the path differs from the same computation in 64 bits (relative 2-norm, largest entry): 7e-7 and
    1.4e-5 on the fp32 kernels, 2.1e-3 and 1e-2 after 8 blocks of the bf16 tier, 3.6e-3 and 2.1e-2 after 16, 1.4e-2 and
    8.5e-2 after 64, 1.1e-2 and 7e-2 after 4 blocks with MXFP8 operands, 6.4e-3 and 8.5e-2 after the MSA module."""
    kind = case["kind"]
    if kind in ("template", "wide", "fold"):
        return {"rel": 5e-6, "max": 1e-4}
    if kind in ("fast", "msa"):
        return {"rel": 2.5e-2 if kind == "msa" else 3e-2, "max": 0.35}
    blocks = case["blocks"]
    rel = 1e-2 if blocks <= 8 else 1.5e-2 if blocks <= 16 else 3e-2
    return {"rel": rel, "max": 12 * rel}
