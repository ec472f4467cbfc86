"""Host-side weight packing for the b200pf kernels.

Input: the reference's flat state dict for one layer (keys as in tt_bio/reference.py:825-863).
Output: device tensors in the layouts include/b200pf.h documents: bf16 rows grouped the way one
GEMM of a kernel wants them, the 0.5 of sigmoid(x) = 0.5 + 0.5 tanh(x / 2) folded into gate rows,
LayerNorm gains / offsets as fp32 vectors the kernels apply themselves.
"""
from __future__ import annotations

import contextlib
import math
from typing import Dict

import torch

from . import _lib

LOG2E = 1.4426950408889634
C_Z = 128
TRI_HEADS, TRI_HEAD_DIM = 4, 32


def pack_trimul(sd: Dict[str, torch.Tensor], pre: str, device) -> Dict[str, torch.Tensor]:
    f = {k: sd[pre + k].detach().to(device=device, dtype=torch.float32) for k in
         ("norm_in.weight", "norm_in.bias", "p_in.weight", "g_in.weight", "norm_out.weight", "norm_out.bias",
          "p_out.weight", "g_out.weight")}
    d = f["p_in.weight"].shape[0] // 2
    if d != C_Z or f["p_in.weight"].shape[1] != C_Z:
        raise RuntimeError("the fused triangle-multiplication kernels are built for c_z = hidden = 128")
    # producer: 0.5 * [p_a | g_a | p_b | g_b], 128 rows each, LayerNorm affine applied in the kernel
    w_pg_tc = 0.5 * torch.cat([f["p_in.weight"][:d], f["g_in.weight"][:d], f["p_in.weight"][d:], f["g_in.weight"][d:]], 0)
    # epilogue: raw-x GEMM with 0.5 * W_pout * gamma_out, LayerNorm over channels applied after the GEMM
    w_pout_tc = (0.5 * f["p_out.weight"] * f["norm_out.weight"][None, :]).to(torch.bfloat16)
    wsum_tc = w_pout_tc.float().sum(1)
    wb_tc = 0.5 * (f["p_out.weight"] * f["norm_out.bias"][None, :]).sum(1)
    w_gout_tc = 0.5 * f["g_out.weight"]
    bf = lambda t: t.to(device=device, dtype=torch.bfloat16).contiguous()
    fp = lambda t: t.to(device=device, dtype=torch.float32).contiguous()
    return {"w_pg_tc": bf(w_pg_tc), "w_pout_tc": bf(w_pout_tc), "wsum_tc": fp(wsum_tc), "wb_tc": fp(wb_tc),
            "w_gout_tc": bf(w_gout_tc), "ln_in_gamma": fp(f["norm_in.weight"]), "ln_in_beta": fp(f["norm_in.bias"])}


def pack_triatt(sd: Dict[str, torch.Tensor], pre: str, device) -> Dict[str, torch.Tensor]:
    f = {k: sd[pre + k].detach().to(device=device, dtype=torch.float32) for k in
         ("layer_norm.weight", "layer_norm.bias", "linear.weight", "mha.linear_q.weight", "mha.linear_k.weight",
          "mha.linear_v.weight", "mha.linear_g.weight", "mha.linear_o.weight")}
    if f["linear.weight"].shape != (TRI_HEADS, C_Z) or f["mha.linear_q.weight"].shape != (TRI_HEADS * TRI_HEAD_DIM, C_Z):
        raise RuntimeError("the fused triangle-attention kernels are built for c_z = 128 and 4 heads x 32")
    # producer: [q (scaled) | k | 0.5 g | v], LayerNorm affine and the bias heads applied in fp32 in the kernel
    w_tc = torch.cat([f["mha.linear_q.weight"] * (LOG2E / math.sqrt(TRI_HEAD_DIM)), f["mha.linear_k.weight"],
                      0.5 * f["mha.linear_g.weight"], f["mha.linear_v.weight"]], 0)
    return {"w_qkgv_tc": w_tc.to(device=device, dtype=torch.bfloat16).contiguous(),
            "w_bias_f32": (f["linear.weight"] * LOG2E).to(device=device, dtype=torch.float32).contiguous(),
            "ln_gamma": f["layer_norm.weight"].to(device=device, dtype=torch.float32).contiguous(),
            "ln_beta": f["layer_norm.bias"].to(device=device, dtype=torch.float32).contiguous(),
            "w_o": f["mha.linear_o.weight"].to(device=device, dtype=torch.bfloat16).contiguous()}


def pack_transition_z(sd: Dict[str, torch.Tensor], pre: str, device) -> Dict[str, torch.Tensor]:
    f = {k: sd[pre + k].detach().to(device=device, dtype=torch.float32) for k in ("norm.weight", "norm.bias", "fc1.weight", "fc2.weight", "fc3.weight")}
    hidden = f["fc1.weight"].shape[0]
    if hidden != 4 * C_Z or f["fc1.weight"].shape[1] != C_Z:
        raise RuntimeError("the fused transition kernel is built for 128 -> 512 -> 128")
    w3 = torch.stack([f["fc3.weight"][:, st * 64:(st + 1) * 64] for st in range(hidden // 64)], 0)   # [8][128][64]
    # per 64-channel chunk [0.5 * fc1 rows | fc2 rows], LayerNorm affine applied in the kernel
    w12_tc = torch.stack([torch.cat([0.5 * f["fc1.weight"][c * 64:(c + 1) * 64], f["fc2.weight"][c * 64:(c + 1) * 64]], 0)
                          for c in range(hidden // 64)], 0)
    return {"w3": w3.to(device=device, dtype=torch.bfloat16).contiguous(),
            "w12_tc": w12_tc.to(device=device, dtype=torch.bfloat16).contiguous(),
            "ln_gamma": f["norm.weight"].to(device=device, dtype=torch.float32).contiguous(),
            "ln_beta": f["norm.bias"].to(device=device, dtype=torch.float32).contiguous()}


def to_device_f32(sd: Dict[str, torch.Tensor], pre: str, device) -> Dict[str, torch.Tensor]:
    """fp32 device copies of every tensor under ``pre`` (keys relative to ``pre``)."""
    return {k[len(pre):]: v.detach().to(device=device, dtype=torch.float32).contiguous()
            for k, v in sd.items() if k.startswith(pre)}


# ------------------------------------------------------------------------------------------------
# fp32-accurate path: weights as 16-bit parts (layouts in include/b200pf.h)
# ------------------------------------------------------------------------------------------------
SPLIT_WIDTHS = (64, 128, 256)
_F16_TARGET = 2.0 ** 14             # scaled values stay at or below this, a factor of four inside fp16's range


def _pow2_scale(bound: float, most: int = 100) -> float:
    """Largest power of two (within 2^-most .. 2^most) that keeps ``bound`` at or below the fp16 target."""
    if not (bound > 0.0 and math.isfinite(bound)):
        return 1.0
    return 2.0 ** max(-most, min(most, math.floor(math.log2(_F16_TARGET / bound))))


QK_MOST = 30        # of a factor whose products stay scaled in the accumulator: times both scales they stay far inside fp32's range


class Versions:
    """Tells whether any of the tensors was changed in place (by an operation that counts versions: one through ``.data`` does not,
    nor do inference tensors)."""

    def __init__(self, tensors) -> None:
        self.tensors = [t for t in tensors if not t.is_inference()]
        self.seen = [t._version for t in self.tensors]

    def changed(self) -> bool:
        return [t._version for t in self.tensors] != self.seen


@contextlib.contextmanager
def packing(device: torch.device, replaced):
    """Around a module's packing, which is over when this is left, so that a later call may read the pack on any stream.  ``replaced``
    is the device of a pack that is dropped for it (or None): kernels of any stream may still read that one, so they are waited for
    too.  Under capture the packing runs at once, on a stream of its own, and not at every replay (nothing is dropped there)."""
    if device.type != "cuda":
        yield
        return
    with torch.cuda.device(device):
        if torch.cuda.is_current_stream_capturing():
            other = torch.cuda.Stream()
            if other == torch.cuda.current_stream():        # streams come from a pool
                other = torch.cuda.Stream()
            with _lib.relaxed_capture(), torch.cuda.stream(other):
                yield
                other.synchronize()
            return
        yield
        torch.cuda.current_stream().synchronize()
    if replaced is not None and replaced.type == "cuda":
        torch.cuda.synchronize(replaced)


class SplitPack:
    """Device tensors of one packed layer and the C structure that points at them."""

    def __init__(self, struct, tensors) -> None:
        self.struct, self.tensors = struct, tensors


def bf16_parts(w: torch.Tensor, device) -> torch.Tensor:
    """[3][...] bf16 parts whose sum is the fp32 value."""
    v = w.detach().float()
    h = v.bfloat16()
    m = (v - h.float()).bfloat16()
    return torch.stack([h, m, (v - h.float() - m.float()).bfloat16()]).to(device).contiguous()


class _Plan:
    """One sub-operation's tensors, the buffer its pack goes to and what is to be written there.

    A plan's builder is a generator: it yields the tensors whose bounds it wants, (weight, None) or (LayerNorm gain, offset), gets for
    each (largest entry, largest 2-norm of a row, bound of a normalised row's entries) and returns the C structure.  So the bounds of
    all sub-operations of a layer are one launch and one synchronisation, and the parts another launch."""

    def __init__(self, sd, pres, device) -> None:
        self.f = {k: v.detach().to(device=device, dtype=torch.float32).contiguous() for k, v in sd.items() if k.startswith(pres)}
        self.buf = torch.empty(sum(_padded(4 * t.numel()) for t in self.f.values()) + _padded(16 * max(t.shape[0] for t in self.f.values())),
                               dtype=torch.uint8, device=device)
        self.used, self.items = 0, []

    def _take(self, nbytes: int) -> int:
        at = self.buf.data_ptr() + self.used
        self.used += _padded(nbytes)
        assert self.used <= self.buf.numel()
        return at

    def vector(self, t: torch.Tensor, scale: float = 1.0, factor: float = 1.0, zeros: int = 0) -> int:
        """fp32 values times factor and scale, and ``zeros`` zeros behind them."""
        at = self._take(4 * (t.numel() + zeros))
        self.items.append(_lib.PackItem(t.data_ptr(), at, 0, 1, t.numel(), 0, factor, scale, 0, 0))
        if zeros:
            self.items.append(_lib.PackItem(None, at + 4 * t.numel(), 0, 1, zeros, 0, 1.0, 1.0, 0, 0))
        return at

    def norm(self, gamma: torch.Tensor, beta: torch.Tensor, scale: float):
        """Pointers of gain and offset times the planes' scale."""
        return self.vector(gamma, scale), self.vector(beta, scale)

    def weight(self, pieces, amax: float, operand_scale: float, interleave: bool = False):
        """SplitWeight of the pieces' rows [(w[rows][k], factor)], one below the other or in turns of 32, for an operand that was
        multiplied by ``operand_scale``."""
        scale, k = _pow2_scale(amax), pieces[0][0].shape[1]
        rows = sum(w.shape[0] for w, _ in pieces)
        at, row0 = self._take(4 * rows * k), 0
        for w, factor in pieces:
            self.items.append(_lib.PackItem(w.data_ptr(), at, rows * k, w.shape[0], k, row0, factor, scale, 2, int(interleave)))
            row0 += 32 if interleave else w.shape[0]
        return _lib.SplitWeight(at, 1.0 / (scale * operand_scale))


def _padded(nbytes: int) -> int:
    return (nbytes + 255) // 256 * 256


def _measure(wanted, device):
    """A float triple per (tensor, offset or None); one synchronisation for all of them."""
    items = [_lib.StatItem(t.data_ptr(), None if b is None else b.data_ptr(), t.numel() // t.shape[-1], t.shape[-1]) for t, b in wanted]
    out = torch.empty(len(items), 3, dtype=torch.float32, device=device)
    _lib.call("b200pf_weight_stats", (_lib.StatItem * len(items))(*items), len(items), out.data_ptr(), _lib.stream())
    return out.tolist()


def pack_split(builders, device):
    """SplitPacks of the builders' sub-operations (made by split_trimul, split_triatt, split_transition, split_single)."""
    builders = list(builders)
    if torch.device(device).type != "cuda":
        raise RuntimeError("part planes are packed on the GPU (there is no CPU path)")
    wanted = [next(b) for _, b in builders]
    values, packs, items = iter(_measure([w for ws in wanted for w in ws], device)), [], []
    for (plan, b), ws in zip(builders, wanted):
        try:
            b.send([next(values) for _ in ws])
        except StopIteration as done:
            packs.append(SplitPack(done.value, [plan.buf]))
        items += plan.items
    _lib.call("b200pf_pack_parts", (_lib.PackItem * len(items))(*items), len(items), _lib.stream())
    return packs


def _builder(build):
    """build(plan, ...) as (plan, generator) of a state dict's sub-operation."""
    def make(sd, pres, device, *args):
        plan = _Plan(sd, pres, device)
        return plan, build(plan, *args)
    return make


def _row_norm(gamma, beta, c: int) -> float:
    """Bound of a normalised row's 2-norm, from the triples of gain and offset."""
    return math.sqrt(c) * gamma[0] + beta[1]


@_builder
def split_trimul(plan, pre: str):
    f = {k[len(pre):]: v for k, v in plan.f.items()}
    gi, bi, go, bo = f["norm_in.weight"], f["norm_in.bias"], f["norm_out.weight"], f["norm_out.bias"]
    p_in, g_in, p_out, g_out = f["p_in.weight"], f["g_in.weight"], f["p_out.weight"], f["g_out.weight"]
    ln_in, off, ln_out, pi, gg, po, gq = yield [(gi, bi), (bi, None), (go, bo), (p_in, None), (g_in, None), (p_out, None), (g_out, None)]
    c = gi.numel()
    s_in, s_out = _pow2_scale(ln_in[2]), _pow2_scale(ln_out[2])
    return _lib.SplitTriMulWeights(*plan.norm(gi, bi, s_in), plan.weight([(p_in, 1.0), (g_in, 1.0)], max(pi[0], gg[0]), s_in), *plan.norm(go, bo, s_out),
                                   plan.weight([(p_out, 1.0)], po[0], s_out), plan.weight([(g_out, 1.0)], gq[0], s_in),
                                   _pow2_scale(pi[1] * _row_norm(ln_in, off, c), QK_MOST), c)


@_builder
def split_triatt(plan, pre: str):
    f = {k[len(pre):]: v for k, v in plan.f.items()}
    g, b, head = f["layer_norm.weight"], f["layer_norm.bias"], f["linear.weight"]
    qw, kw, vw, gw, ow = (f[f"mha.linear_{x}.weight"] for x in "qkvgo")
    heads, c = head.shape
    hd = qw.shape[0] // heads
    qs = LOG2E / math.sqrt(hd)
    ln, off, sq, sk, sv, sg, so = yield [(g, b), (b, None), (qw, None), (kw, None), (vw, None), (gw, None), (ow, None)]
    norm = _row_norm(ln, off, c)
    s_in, o_scale = _pow2_scale(ln[2]), _pow2_scale(sv[1] * norm)         # an attention output is an average of rows of v
    return _lib.SplitTriAttWeights(*plan.norm(g, b, s_in), plan.vector(head, 1.0 / s_in, LOG2E),
                                   plan.weight([(qw, qs), (kw, 1.0), (vw, 1.0), (gw, 1.0)], max(qs * sq[0], sk[0], sv[0], sg[0]), s_in),
                                   plan.weight([(ow, 1.0)], so[0], o_scale), o_scale, _pow2_scale(qs * sq[1] * norm, QK_MOST),
                                   _pow2_scale(sk[1] * norm, QK_MOST), c, heads, hd)


def _swiglu_wanted(f):
    g, b = f["norm.weight"], f["norm.bias"]
    return [(g, b), (b, None), (f["fc1.weight"], None), (f["fc2.weight"], None), (f["fc3.weight"], None)]


def _swiglu(plan, f, values):
    """(gain, offset), fc12, fc3, hidden scale; |silu(a) b| <= |a| |b|.  fc12: 32 rows of fc1, then 32 of fc2, in turn, so that a
    64-column block of the product holds both factors of 32 hidden channels."""
    ln, off, s1, s2, s3 = values
    norm = _row_norm(ln, off, f["norm.weight"].numel())
    s_in, hs = _pow2_scale(ln[2]), _pow2_scale(s1[1] * norm * s2[1] * norm)
    return (plan.norm(f["norm.weight"], f["norm.bias"], s_in),
            plan.weight([(f["fc1.weight"], 1.0), (f["fc2.weight"], 1.0)], max(s1[0], s2[0]), s_in, interleave=True),
            plan.weight([(f["fc3.weight"], 1.0)], s3[0], hs), hs)


@_builder
def split_transition(plan, pre: str):
    f = {k[len(pre):]: v for k, v in plan.f.items()}
    values = yield _swiglu_wanted(f)
    gb, fc12, fc3, hs = _swiglu(plan, f, values)
    return _lib.SplitTransitionWeights(*gb, fc12, fc3, hs, f["norm.weight"].numel(), f["fc1.weight"].shape[0])


@_builder
def split_single(plan, pre: str, num_heads: int):
    """pre_norm_s, attention (without the pair-bias projection) and transition_s of one layer."""
    f = {k[len(pre):]: v for k, v in plan.f.items()}
    t = {k[len("transition_s."):]: v for k, v in f.items() if k.startswith("transition_s.")}
    g, b, bias = f["pre_norm_s.weight"], f["pre_norm_s.bias"], f["attention.proj_q.bias"]
    qw, kw, vw, gw, ow = (f[f"attention.proj_{x}.weight"] for x in "qkvgo")
    cs = g.numel()
    qs = LOG2E / math.sqrt(cs // num_heads)
    ln, off, sq, sk, sv, sg, so, sb, *values = yield [(g, b), (b, None), (qw, None), (kw, None), (vw, None), (gw, None), (ow, None), (bias, None),
                                                      *_swiglu_wanted(t)]
    norm = _row_norm(ln, off, cs)
    s_in, o_scale = _pow2_scale(ln[2]), _pow2_scale(sv[1] * norm)
    ln_ptrs = plan.norm(g, b, s_in)
    w_qkvg = plan.weight([(qw, qs), (kw, 1.0), (vw, 1.0), (gw, 1.0)], max(qs * sq[0], sk[0], sv[0], sg[0]), s_in)
    bias_ptr, w_o = plan.vector(bias, 1.0, qs, zeros=3 * cs), plan.weight([(ow, 1.0)], so[0], o_scale)
    gb, fc12, fc3, hs = _swiglu(plan, t, values)
    return _lib.SingleTrackWeights(*ln_ptrs, w_qkvg, bias_ptr, w_o, o_scale, _pow2_scale(qs * (sq[1] * norm + sb[0]), QK_MOST),
                                   _pow2_scale(sk[1] * norm, QK_MOST), *gb, fc12, hs, fc3, cs, num_heads, t["fc1.weight"].shape[0])


def pack_split_trimul(sd, pre: str, device) -> SplitPack:
    return pack_split([split_trimul(sd, pre, device, pre)], device)[0]


def pack_split_triatt(sd, pre: str, device) -> SplitPack:
    return pack_split([split_triatt(sd, pre, device, pre)], device)[0]


def pack_split_transition(sd, pre: str, device) -> SplitPack:
    return pack_split([split_transition(sd, pre, device, pre)], device)[0]


def single_builder(sd, pre: str, num_heads: int, device):
    # proj_z, the pair-bias projection, is packed by pack_pair_bias
    own = {k: v for k, v in sd.items() if not k.startswith(pre + "attention.proj_z.")}
    return split_single(own, (pre + "pre_norm_s.", pre + "attention.", pre + "transition_s."), device, pre, num_heads)


def pack_pair_bias(sd, pre: str, device) -> Dict[str, torch.Tensor]:
    """The single track's only read of z: LayerNorm and the head projection, in the base-2 logarithms the attention works in."""
    f = {k[len(pre):]: v.detach().to(device=device, dtype=torch.float32) for k, v in sd.items() if k.startswith(pre)}
    fp = lambda t: t.to(device=device, dtype=torch.float32).contiguous()
    return {"gamma": fp(f["proj_z.0.weight"]), "beta": fp(f["proj_z.0.bias"]), "w": fp(f["proj_z.1.weight"] * LOG2E)}
