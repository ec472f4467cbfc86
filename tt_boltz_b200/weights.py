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


def _f16_parts(w: torch.Tensor, scale: float) -> torch.Tensor:
    v = w * scale                       # exact: a power of two
    hi = v.half()
    return torch.stack([hi, (v - hi.float()).half()])


def bf16_parts(w: torch.Tensor, device) -> torch.Tensor:
    """[3][...] bf16 parts whose sum is the fp32 value."""
    v = w.detach().float()
    h = v.bfloat16()
    m = (v - h.float()).bfloat16()
    return torch.stack([h, m, (v - h.float() - m.float()).bfloat16()]).to(device).contiguous()


def _fetch(**values: torch.Tensor) -> Dict[str, float]:
    """Device scalars as host numbers, one synchronisation for all of them."""
    return dict(zip(values, torch.stack([v.reshape(()).float() for v in values.values()]).tolist()))


def _ln_bound(gamma: torch.Tensor, beta: torch.Tensor) -> torch.Tensor:
    """Bound of a normalised row's entries."""
    return (math.sqrt(gamma.numel()) * gamma.abs() + beta.abs()).max()


def _row_norm(gamma: torch.Tensor, beta: torch.Tensor) -> torch.Tensor:
    """Bound of a normalised row's 2-norm."""
    return math.sqrt(gamma.numel()) * gamma.abs().max() + beta.norm()


def _projection_bound(w: torch.Tensor, row_norm: torch.Tensor) -> torch.Tensor:
    """Bound of |x w^T| for rows x of at most that 2-norm."""
    return w.norm(dim=1).max() * row_norm


def _split_weight(keep, w: torch.Tensor, amax: float, operand_scale: float):
    """SplitWeight of w[n][k] for an operand that was multiplied by ``operand_scale``; its tensor is appended to ``keep``."""
    from ._lib import SplitWeight
    scale = _pow2_scale(amax)
    keep.append(_f16_parts(w, scale))
    return SplitWeight(keep[-1].data_ptr(), 1.0 / (scale * operand_scale))


def _ln(keep, gamma: torch.Tensor, beta: torch.Tensor, scale: float):
    """Pointers of gain and offset times the planes' scale."""
    keep += [gamma * scale, beta * scale]
    return keep[-2].data_ptr(), keep[-1].data_ptr()


def _on(sd, pre, device):
    return {k[len(pre):]: v.detach().to(device=device, dtype=torch.float32) for k, v in sd.items() if k.startswith(pre)}


def _swiglu_rows(fc1: torch.Tensor, fc2: torch.Tensor) -> torch.Tensor:
    """32 rows of fc1, then 32 of fc2, in turn: a 64-column block of the product holds both factors of 32 hidden channels."""
    h, k = fc1.shape
    return torch.stack([fc1.view(h // 32, 32, k), fc2.view(h // 32, 32, k)], 1).reshape(2 * h, k)


def pack_split_trimul(sd, pre: str, device):
    from ._lib import SplitTriMulWeights
    f, keep = _on(sd, pre, device), []
    w_in = torch.cat([f["p_in.weight"], f["g_in.weight"]], 0)
    gi, bi, go, bo = f["norm_in.weight"], f["norm_in.bias"], f["norm_out.weight"], f["norm_out.bias"]
    v = _fetch(ln_in=_ln_bound(gi, bi), ln_out=_ln_bound(go, bo), w_in=w_in.abs().max(), p=f["p_out.weight"].abs().max(),
               g=f["g_out.weight"].abs().max(), u=_projection_bound(f["p_in.weight"], _row_norm(gi, bi)))
    s_in, s_out = _pow2_scale(v["ln_in"]), _pow2_scale(v["ln_out"])
    st = SplitTriMulWeights(*_ln(keep, gi, bi, s_in), _split_weight(keep, w_in, v["w_in"], s_in), *_ln(keep, go, bo, s_out),
                            _split_weight(keep, f["p_out.weight"], v["p"], s_out), _split_weight(keep, f["g_out.weight"], v["g"], s_in),
                            _pow2_scale(v["u"], QK_MOST), gi.numel())
    return SplitPack(st, keep)


def pack_split_triatt(sd, pre: str, device):
    from ._lib import SplitTriAttWeights
    f, keep = _on(sd, pre, device), []
    heads, c = f["linear.weight"].shape
    hd = f["mha.linear_q.weight"].shape[0] // heads
    g, b = f["layer_norm.weight"], f["layer_norm.bias"]
    qkvg = torch.cat([f["mha.linear_q.weight"] * (LOG2E / math.sqrt(hd)), f["mha.linear_k.weight"], f["mha.linear_v.weight"],
                      f["mha.linear_g.weight"]], 0)
    norm, ht = _row_norm(g, b), heads * hd
    v = _fetch(ln=_ln_bound(g, b), w=qkvg.abs().max(), o=f["mha.linear_o.weight"].abs().max(),
               q=_projection_bound(qkvg[:ht], norm), k=_projection_bound(qkvg[ht:2 * ht], norm), v=_projection_bound(qkvg[2 * ht:3 * ht], norm))
    s_in, o_scale = _pow2_scale(v["ln"]), _pow2_scale(v["v"])       # an attention output is an average of rows of v
    ln = _ln(keep, g, b, s_in)
    keep.append((f["linear.weight"] * (LOG2E / s_in)).contiguous())
    st = SplitTriAttWeights(*ln, keep[-1].data_ptr(), _split_weight(keep, qkvg, v["w"], s_in),
                            _split_weight(keep, f["mha.linear_o.weight"], v["o"], o_scale), o_scale, _pow2_scale(v["q"], QK_MOST),
                            _pow2_scale(v["k"], QK_MOST), c, heads, hd)
    return SplitPack(st, keep)


def _swiglu_stats(f) -> Dict[str, torch.Tensor]:
    """|silu(a) b| <= |a| |b|."""
    g, b = f["norm.weight"], f["norm.bias"]
    norm = _row_norm(g, b)
    return {"t_ln": _ln_bound(g, b), "t_h": _projection_bound(f["fc1.weight"], norm) * _projection_bound(f["fc2.weight"], norm),
            "t_12": torch.maximum(f["fc1.weight"].abs().max(), f["fc2.weight"].abs().max()), "t_3": f["fc3.weight"].abs().max()}


def _pack_swiglu(f, keep, v):
    """(gain, offset), fc12, fc3, hidden scale."""
    s_in, hs = _pow2_scale(v["t_ln"]), _pow2_scale(v["t_h"])
    return (_ln(keep, f["norm.weight"], f["norm.bias"], s_in),
            _split_weight(keep, _swiglu_rows(f["fc1.weight"], f["fc2.weight"]), v["t_12"], s_in),
            _split_weight(keep, f["fc3.weight"], v["t_3"], hs), hs)


def pack_split_transition(sd, pre: str, device):
    from ._lib import SplitTransitionWeights
    f, keep = _on(sd, pre, device), []
    gb, fc12, fc3, hs = _pack_swiglu(f, keep, _fetch(**_swiglu_stats(f)))
    return SplitPack(SplitTransitionWeights(*gb, fc12, fc3, hs, f["norm.weight"].numel(), f["fc1.weight"].shape[0]), keep)


def pack_single_track(sd, pre: str, num_heads: int, device):
    """Single track: pre_norm_s, attention (without the pair-bias projection) and transition_s of one layer."""
    from ._lib import SingleTrackWeights
    keep = []
    n, a, t = (_on(sd, pre + part, device) for part in ("pre_norm_s.", "attention.", "transition_s."))
    g, b, cs = n["weight"], n["bias"], n["weight"].numel()
    qs = LOG2E / math.sqrt(cs // num_heads)
    qkvg = torch.cat([a["proj_q.weight"] * qs, a["proj_k.weight"], a["proj_v.weight"], a["proj_g.weight"]], 0)
    norm = _row_norm(g, b)
    v = _fetch(ln=_ln_bound(g, b), w=qkvg.abs().max(), o=a["proj_o.weight"].abs().max(),
               q=_projection_bound(qkvg[:cs], norm) + (a["proj_q.bias"] * qs).abs().max(), k=_projection_bound(qkvg[cs:2 * cs], norm),
               v=_projection_bound(a["proj_v.weight"], norm), **_swiglu_stats(t))
    s_in, o_scale = _pow2_scale(v["ln"]), _pow2_scale(v["v"])
    ln = _ln(keep, g, b, s_in)
    keep.append(torch.nn.functional.pad(a["proj_q.bias"] * qs, (0, 3 * cs)))
    bias = keep[-1].data_ptr()
    w_qkvg, w_o = _split_weight(keep, qkvg, v["w"], s_in), _split_weight(keep, a["proj_o.weight"], v["o"], o_scale)
    gb2, fc12, fc3, hs = _pack_swiglu(t, keep, v)
    return SplitPack(SingleTrackWeights(*ln, w_qkvg, bias, w_o, o_scale, _pow2_scale(v["q"], QK_MOST), _pow2_scale(v["k"], QK_MOST), *gb2, fc12, hs, fc3, cs, num_heads, t["fc1.weight"].shape[0]), keep)


def pack_pair_bias(sd, pre: str, device) -> Dict[str, torch.Tensor]:
    """The single track's only read of z: LayerNorm and the head projection, in the base-2 logarithms the attention works in."""
    f = _on(sd, pre, device)
    fp = lambda t: t.to(device=device, dtype=torch.float32).contiguous()
    return {"gamma": fp(f["proj_z.0.weight"]), "beta": fp(f["proj_z.0.bias"]), "w": fp(f["proj_z.1.weight"] * LOG2E)}
