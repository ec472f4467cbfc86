"""Host orchestration of the Pairformer sub-operations on one GPU.

Each function enqueues b200pf kernels (through the C ABI) on torch's current stream and updates
the fp32 residual tensor in place.  Tensors here are B = 1 folded away: z [N, N, 128] fp32,
s [N, 384] fp32, masks uint8.  Nothing in this file computes on the CPU or with torch math.
"""
from __future__ import annotations

import ctypes as C
import math
from typing import Dict, Optional

import torch

from . import _lib, weights
from ._lib import PlaneOut, Planes, call, ptr, stream

C_Z = 128


def _round_up(x: int, m: int) -> int:
    return (x + m - 1) // m * m


class PairMasks:
    """uint8 forms of the pair mask: [N][N] for the triangle multiplication, and one contiguous,
    64-padded row per attention line for the starting (rows) and ending (columns) node."""

    def __init__(self, pair_mask_u8: torch.Tensor) -> None:
        n = pair_mask_u8.shape[0]
        self.n = n
        self.pitch = _round_up(n, 64)
        self.pm = pair_mask_u8.contiguous()
        self.rows = torch.zeros(n, self.pitch, dtype=torch.uint8, device=pair_mask_u8.device)
        self.rows[:, :n] = self.pm
        self.cols = torch.zeros(n, self.pitch, dtype=torch.uint8, device=pair_mask_u8.device)
        self.cols[:, :n] = self.pm.t()

    def scratch(self, ws: "Workspace") -> _lib.PairScratch:
        """The workspace and the masks as ``b200pf_pair_block`` takes them."""
        return _lib.PairScratch((C.c_void_p * 5)(*[ptr(b) for b in ws.buf]), ptr(ws.tri_bias), ptr(self.pm), ptr(self.rows), ptr(self.cols), ws.n, ws.pitch,
                                self.pitch)


# Rows of planes start on 64-byte boundaries, so that a 128-byte box of one touches four 32-byte sectors and no half-written one.  With rows of
# a multiple of 8 elements, 16 bytes off a sector at every other size, a block of the bf16 tier took 1972 us for 1916 at 600 tokens, 5335
# for 5173 at 900, 409.0 for 401.5 at 264, 154.8 for 152.9 at 136 and 114.1 for 112.8 at 117; on 32-byte boundaries 836.6 for 822.7 at 400.
PLANE_PITCH = 32


class Workspace:
    """bf16 scratch for one token count: five [N*pitch*128] buffers shared by the sub-operations
    (triangle multiplication uses three as a / b / x planes, triangle attention five as
    q / k / v / g / o), plus the triangle-bias tile source [4][N][pitch]."""

    def __init__(self, n: int, device) -> None:
        self.n = n
        self.pitch = _round_up(n, PLANE_PITCH)
        self.plane_stride = n * self.pitch
        elems = C_Z * self.plane_stride
        self.buf = [torch.empty(elems, dtype=torch.bfloat16, device=device) for _ in range(5)]
        self.tri_bias = torch.empty(4 * n * self.pitch, dtype=torch.bfloat16, device=device)
        self._mx_scales = None

    def mx_scales(self):
        """Two zero-initialised e8m0 scale buffers (a and b operand) for the MXFP8 triangle multiplication."""
        if self._mx_scales is None:
            nbytes = _lib.load().b200pf_mx_scale_bytes(self.n, self.n, C_Z)
            self._mx_scales = [torch.zeros(nbytes, dtype=torch.uint8, device=self.buf[0].device) for _ in range(2)]
        return self._mx_scales


# ------------------------------------------------------------------------------------------------
# bf16 tier (fused kernels)
# ------------------------------------------------------------------------------------------------
def trimul_producer_weights(w: Dict[str, torch.Tensor]):
    """(ln_gamma, ln_beta, w_pg) pointers of the triangle-multiplication producer."""
    return ptr(w["ln_in_gamma"]), ptr(w["ln_in_beta"]), ptr(w["w_pg_tc"])


def triatt_producer_weights(w: Dict[str, torch.Tensor]):
    """(ln_gamma, ln_beta, w_bias_f32, w_qkgv) pointers of the triangle-attention producer."""
    return ptr(w["ln_gamma"]), ptr(w["ln_beta"]), ptr(w["w_bias_f32"]), ptr(w["w_qkgv_tc"])


def trimul_epilogue(z, x, plane_stride, pitch, w, rows, n) -> None:
    call("b200pf_trimul_epilogue_tc", ptr(z), ptr(x), plane_stride, pitch, ptr(w["ln_in_gamma"]), ptr(w["ln_in_beta"]),
         ptr(w["w_pout_tc"]), ptr(w["w_gout_tc"]), ptr(w["wsum_tc"]), ptr(w["wb_tc"]), rows, n, stream())


def tri_mul_bf16(z: torch.Tensor, mask_u8: torch.Tensor, w: Dict[str, torch.Tensor], ws: Workspace,
                 incoming: bool) -> None:
    n = z.shape[0]
    a, b, x = ws.buf[0], ws.buf[1], ws.buf[2]
    st = stream()
    oa = PlaneOut(ptr(a), ws.plane_stride, 0, 0)
    ob = PlaneOut(ptr(b), ws.plane_stride, 0, 0)
    call("b200pf_trimul_producer", ptr(z), ptr(mask_u8), *trimul_producer_weights(w), C.byref(oa), C.byref(ob),
         ws.pitch, n, n, int(incoming), st)
    pa = Planes(ptr(a), ws.plane_stride, 0, ws.pitch, n, n, 1, 0)
    pb = Planes(ptr(b), ws.plane_stride, 0, ws.pitch, n, n, 1, 0)
    call("b200pf_trimul_contract", C.byref(pa), C.byref(pb), None, None, ptr(x), ws.plane_stride, ws.pitch,
         0, 0, C_Z, 0, st)
    trimul_epilogue(z, x, ws.plane_stride, ws.pitch, w, n, n)


def tri_mul_mxfp8(z: torch.Tensor, mask_u8: torch.Tensor, w: Dict[str, torch.Tensor], ws: Workspace,
                  incoming: bool, contract_variant: int = 2) -> None:
    """Triangle multiplication with MXFP8 operands (e4m3 values, e8m0 scale per 32 along k).

    contract_variant 2 = block-scaled tcgen05 contraction; 0 = expand the operands to bf16
    (exactly) and run the bf16 contraction: the cross-check of variant 2.
    """
    n = z.shape[0]
    st = stream()
    pitch8 = _round_up(n, 2 * PLANE_PITCH)
    stride8 = n * pitch8
    a8, b8 = ws.buf[3].view(torch.uint8), ws.buf[4].view(torch.uint8)
    sa, sb = ws.mx_scales()
    x = ws.buf[2]
    call("b200pf_trimul_producer_mx", ptr(z), ptr(mask_u8), ptr(w["ln_in_gamma"]), ptr(w["ln_in_beta"]), ptr(w["w_pg_tc"]),
         ptr(a8), ptr(b8), ptr(sa), ptr(sb), stride8, pitch8, n, n, int(incoming), st)
    if contract_variant == 2:
        pa = Planes(ptr(a8), stride8, 0, pitch8, n, n, 1, 0)
        pb = Planes(ptr(b8), stride8, 0, pitch8, n, n, 1, 0)
        call("b200pf_trimul_contract", C.byref(pa), C.byref(pb), ptr(sa), ptr(sb), ptr(x), ws.plane_stride, ws.pitch, 0, 0, C_Z, 2, st)
    else:
        a, b = ws.buf[0], ws.buf[1]
        for src, sc, dst in ((a8, sa, a), (b8, sb, b)):
            call("b200pf_mx_dequant", ptr(src), ptr(sc), ptr(dst), stride8, pitch8, ws.plane_stride, ws.pitch, n, n, C_Z, st)
        pa = Planes(ptr(a), ws.plane_stride, 0, ws.pitch, n, n, 1, 0)
        pb = Planes(ptr(b), ws.plane_stride, 0, ws.pitch, n, n, 1, 0)
        call("b200pf_trimul_contract", C.byref(pa), C.byref(pb), None, None, ptr(x), ws.plane_stride, ws.pitch,
             0, 0, C_Z, 0, st)
    trimul_epilogue(z, x, ws.plane_stride, ws.pitch, w, n, n)


def tri_att_bf16(z: torch.Tensor, masks: PairMasks, w: Dict[str, torch.Tensor], ws: Workspace, ending: bool) -> None:
    n = z.shape[0]
    q, k, v, g, o = ws.buf
    st = stream()
    bias_hs, bias_qs = ws.pitch, 4 * ws.pitch          # layout [query][head][key]: a row shard is contiguous
    call("b200pf_triatt_producer", ptr(z), *triatt_producer_weights(w), ptr(q), ptr(k), ptr(v), ptr(g),
         ptr(ws.tri_bias), bias_hs, bias_qs, ws.pitch, n, n, int(ending), st)
    if ending:      # line = column j: o element (line, pos) -> z position [pos][line]
        o_ls, o_ps = C_Z, n * C_Z
    else:
        o_ls, o_ps = n * C_Z, C_Z
    lines_mask = masks.cols if ending else masks.rows
    call("b200pf_triatt_core_tc4", ptr(q), ptr(k), ptr(v), ws.pitch, ptr(ws.tri_bias), bias_hs, bias_qs,
         ptr(lines_mask), masks.pitch, ptr(o), o_ls, o_ps, n, n, st)
    call("b200pf_triatt_epilogue", ptr(z), ptr(o), ptr(g), ptr(w["w_o"]), n * n, st)


def transition_z_bf16(z: torch.Tensor, w: Dict[str, torch.Tensor]) -> None:
    rows = z.shape[0] * z.shape[1]
    call("b200pf_transition_z_tc", ptr(z), ptr(w["ln_gamma"]), ptr(w["ln_beta"]), ptr(w["w12_tc"]), ptr(w["w3"]), rows, stream())


class PairBlock:
    """The pair track of one block as a single call: the packed weights of the five sub-operations as the C structure."""

    def __init__(self, pk) -> None:
        mul = lambda w: _lib.TriMulWeights(ptr(w["ln_in_gamma"]), ptr(w["ln_in_beta"]), ptr(w["w_pg_tc"]), ptr(w["w_pout_tc"]), ptr(w["w_gout_tc"]),
                                           ptr(w["wsum_tc"]), ptr(w["wb_tc"]))
        att = lambda w: _lib.TriAttWeights(ptr(w["ln_gamma"]), ptr(w["ln_beta"]), ptr(w["w_bias_f32"]), ptr(w["w_qkgv_tc"]), ptr(w["w_o"]))
        t = pk["transition_z"]
        self.struct = _lib.PairWeights(mul(pk["tri_mul_out"]), mul(pk["tri_mul_in"]), att(pk["tri_att_start"]), att(pk["tri_att_end"]),
                                       _lib.TransitionWeights(ptr(t["ln_gamma"]), ptr(t["ln_beta"]), ptr(t["w12_tc"]), ptr(t["w3"])))

    def run(self, z: torch.Tensor, scratch: _lib.PairScratch) -> None:
        call("b200pf_pair_block", ptr(z), C.byref(self.struct), C.byref(scratch), stream())


# ------------------------------------------------------------------------------------------------
# un-fused fp32 kernels: fp32 tier and single track at widths that the part-plane kernels below are not built for, recycling
# ------------------------------------------------------------------------------------------------
def _empty(rows: int, c: int, like: torch.Tensor) -> torch.Tensor:
    return torch.empty(rows, c, dtype=torch.float32, device=like.device)


def f32_layernorm(x: torch.Tensor, gamma: torch.Tensor, beta: torch.Tensor) -> torch.Tensor:
    rows, c = x.numel() // x.shape[-1], x.shape[-1]
    y = _empty(rows, c, x)
    call("b200pf_f32_layernorm", ptr(x), ptr(gamma), ptr(beta), ptr(y), rows, c, stream())
    return y


def f32_linear(x: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None,
               out: Optional[torch.Tensor] = None, accumulate: bool = False) -> torch.Tensor:
    k = w.shape[1]
    rows = x.numel() // k
    if out is None:
        out = _empty(rows, w.shape[0], x)
    call("b200pf_f32_linear", ptr(x), ptr(w), ptr(bias), ptr(out), rows, k, w.shape[0], int(accumulate), stream())
    return out


def f32_gate(a: torch.Tensor, b: torch.Tensor, mode: int, row_mask: Optional[torch.Tensor] = None,
             out: Optional[torch.Tensor] = None) -> torch.Tensor:
    c = a.shape[-1]
    rows = a.numel() // c
    if out is None:
        out = _empty(rows, c, a)
    call("b200pf_f32_gate", ptr(a), ptr(b), ptr(row_mask), ptr(out), rows, c, mode, stream())
    return out


def tri_mul_f32(z: torch.Tensor, mask_u8: torch.Tensor, w: Dict[str, torch.Tensor], incoming: bool) -> None:
    n = z.shape[0]
    x = f32_layernorm(z, w["norm_in.weight"], w["norm_in.bias"])
    u = f32_gate(f32_linear(x, w["p_in.weight"]), f32_linear(x, w["g_in.weight"]), 0, mask_u8)     # [N*N, 2D]
    d = u.shape[1] // 2
    t = _empty(n * n, d, z)
    call("b200pf_f32_trimul_contract", ptr(u), u.data_ptr() + 4 * d, ptr(t), n, d, 2 * d, int(incoming), stream())
    tn = f32_layernorm(t, w["norm_out.weight"], w["norm_out.bias"])
    f32_gate(f32_linear(tn, w["p_out.weight"]), f32_linear(x, w["g_out.weight"]), 2, out=z)


def _attention_f32(q, k, v, bias, bias_strides, mask_u8, mask_strides, batch, n_q, n_k, heads, hd, rs, ps,
                   scale, inf_value, order) -> torch.Tensor:
    o = torch.empty_like(q)
    call("b200pf_f32_attention", ptr(q), ptr(k), ptr(v), ptr(o), ptr(bias), *bias_strides, ptr(mask_u8),
         *mask_strides, batch, n_q, n_k, heads, hd, rs, ps, scale, inf_value, order, stream())
    return o


def tri_att_f32(z: torch.Tensor, mask_u8: torch.Tensor, w: Dict[str, torch.Tensor], ending: bool) -> None:
    n, c = z.shape[0], z.shape[-1]
    st = stream()
    if ending:      # the reference transposes z and the mask, runs the starting-node path, transposes back
        src = torch.empty_like(z)
        call("b200pf_f32_transpose01", ptr(z), ptr(src), n, c, 0, st)
        mask_ls, mask_ks = 1, n
    else:
        src = z
        mask_ls, mask_ks = n, 1
    heads = w["linear.weight"].shape[0]
    hd = w["mha.linear_q.weight"].shape[0] // heads
    x = f32_layernorm(src, w["layer_norm.weight"], w["layer_norm.bias"])
    bias = torch.empty(heads, n * n, dtype=torch.float32, device=z.device)
    if c == C_Z and heads in (4, 16):       # one fused pass over z
        call("b200pf_ln_proj_heads", ptr(src), ptr(w["layer_norm.weight"]), ptr(w["layer_norm.bias"]),
             ptr(w["linear.weight"]), ptr(bias), n * n, n * n, c, heads, st)
    else:                                   # other widths / head counts: the normalised rows through the transposing linear
        call("b200pf_f32_linear_t", ptr(x), ptr(w["linear.weight"]), None, ptr(bias), n * n, n * n, c, heads, st)
    q = f32_linear(x, w["mha.linear_q.weight"])
    k = f32_linear(x, w["mha.linear_k.weight"])
    v = f32_linear(x, w["mha.linear_v.weight"])
    g = f32_linear(x, w["mha.linear_g.weight"])
    o = _attention_f32(q, k, v, bias, (n * n, n, 1), mask_u8, (mask_ls, mask_ks), n, n, n, heads, hd,
                       n * heads * hd, heads * hd, 1.0 / math.sqrt(hd), 1e9, 0)
    og = f32_gate(o, g, 0)
    if ending:
        upd = f32_linear(og, w["mha.linear_o.weight"])
        call("b200pf_f32_transpose01", ptr(upd), ptr(z), n, c, 1, st)
    else:
        f32_linear(og, w["mha.linear_o.weight"], out=z, accumulate=True)


def transition_f32(x_res: torch.Tensor, w: Dict[str, torch.Tensor]) -> None:
    x = f32_layernorm(x_res, w["norm.weight"], w["norm.bias"])
    h = f32_gate(f32_linear(x, w["fc1.weight"]), f32_linear(x, w["fc2.weight"]), 1)
    f32_linear(h, w["fc3.weight"], out=x_res, accumulate=True)


# ------------------------------------------------------------------------------------------------
# fp32-accurate tensor-core path (16-bit parts): pair track of the fp32 tier, single track of every tier
# ------------------------------------------------------------------------------------------------
class Scratch:
    """A call's workspace: one buffer that grows to the largest request.  Made per call and per stream, never kept, so that
    calls on several streams or threads do not meet in it."""

    def __init__(self, device) -> None:
        self.device, self.buf = device, None

    def get(self, nbytes: int) -> int:
        if self.buf is None or self.buf.numel() < nbytes:
            self.buf = torch.empty(nbytes, dtype=torch.uint8, device=self.device)
        return self.buf.data_ptr()


def _nbytes(name: str, *args) -> int:
    return int(getattr(_lib.load(), name)(*args))


def tri_mul_split(z: torch.Tensor, mask_u8: torch.Tensor, pack, incoming: bool, scratch: Scratch) -> None:
    n = z.shape[0]
    ws = scratch.get(_nbytes("b200pf_split_pair_workspace", n, pack.struct.c, 0, 0, 0))
    call("b200pf_split_tri_mul", ptr(z), ptr(mask_u8), C.byref(pack.struct), n, int(incoming), ws, stream())


def tri_att_split(z: torch.Tensor, mask_u8: torch.Tensor, pack, ending: bool, scratch: Scratch) -> None:
    n, w = z.shape[0], pack.struct
    ws = scratch.get(_nbytes("b200pf_split_pair_workspace", n, w.c, w.heads, w.hd, 0))
    call("b200pf_split_tri_att", ptr(z), ptr(mask_u8), C.byref(w), n, int(ending), ws, stream())


def transition_split(x: torch.Tensor, pack, scratch: Scratch) -> None:
    w, rows = pack.struct, x.numel() // pack.struct.c
    nbytes = _nbytes("b200pf_split_transition_workspace", rows, w.c, w.hidden)
    call("b200pf_split_transition", ptr(x), rows, C.byref(w), scratch.get(nbytes), nbytes, stream())


def split_linear(x: torch.Tensor, w_parts: torch.Tensor, bias: Optional[torch.Tensor], out: torch.Tensor, accumulate: bool, scratch: Scratch) -> None:
    """out (+)= x w^T (+ bias) with ``w_parts`` = weights.bf16_parts(w): any finite fp32 x, all 24 bits of both factors."""
    k, n = w_parts.shape[2], w_parts.shape[1]
    rows = x.numel() // k
    ws = scratch.get(_nbytes("b200pf_split_linear_workspace", rows, k))
    call("b200pf_split_linear", ptr(x), ptr(w_parts), ptr(bias), ptr(out), rows, k, n, int(accumulate), ws, stream())


class SingleTrack:
    """s += AttentionPairBias(LN(s), z); s += Transition(s) in fp32 (tt_bio/reference.py:906-912) of one layer, on part
    planes: ``bias`` (its only read of z), ``attention`` for a range of query rows, ``finish`` per row."""

    def __init__(self, sd, pre: str, num_heads: int, device, pack=None) -> None:
        self.pack = pack or weights.pack_split([weights.single_builder(sd, pre, num_heads, device)], device)[0]
        self.z_bias = weights.pack_pair_bias(sd, pre + "attention.", device)
        b = self.z_bias
        self.bias_struct = _lib.PairBiasWeights(ptr(b["gamma"]), ptr(b["beta"]), ptr(b["w"]), b["w"].shape[1], b["w"].shape[0])

    def bias(self, z_rows: torch.Tensor) -> torch.Tensor:
        """bias[h][i_local * N + j], times log2(e): one fp32 pass over the (local rows of) z [nr, N, c_z]."""
        rows, c = z_rows.shape[0] * z_rows.shape[1], z_rows.shape[-1]
        w = self.z_bias
        heads = w["w"].shape[0]
        out = torch.empty(heads, rows, dtype=torch.float32, device=z_rows.device)
        name = "b200pf_ln_proj_heads" if c == C_Z and heads in (4, 16) else "b200pf_ln_heads"
        call(name, ptr(z_rows), ptr(w["gamma"]), ptr(w["beta"]), ptr(w["w"]), ptr(out), rows, rows, c, heads, stream())
        return out

    def attention(self, s: torch.Tensor, bias: torch.Tensor, tok_mask_u8: Optional[torch.Tensor], r0: int, nq: int, scratch: Scratch) -> torch.Tensor:
        w = self.pack.struct
        og = torch.empty(2, nq, w.cs, dtype=torch.float16, device=s.device)
        ws = scratch.get(_nbytes("b200pf_single_track_workspace", s.shape[0], w.cs, w.hidden))
        call("b200pf_single_track_attention", ptr(s), C.byref(w), ptr(bias), ptr(tok_mask_u8), ptr(og), s.shape[0], r0, nq, ws, stream())
        return og

    def rows(self, s: torch.Tensor, bias: torch.Tensor, tok_mask_u8: Optional[torch.Tensor], scratch: Scratch) -> None:
        """``attention`` and ``finish`` for every row."""
        w, n = self.pack.struct, s.shape[0]
        ws = scratch.get(_nbytes("b200pf_single_track_rows_workspace", n, w.cs, w.hidden))
        call("b200pf_single_track_rows", ptr(s), C.byref(w), ptr(bias), ptr(tok_mask_u8), n, ws, stream())

    def beside(self, s: torch.Tensor, z: torch.Tensor, bias: torch.Tensor, tok_mask_u8: Optional[torch.Tensor], scratch: Scratch, side: int,
               ready: int, done: int, wait_done: bool) -> None:
        """``bias`` into the given buffer on the current stream, ``rows`` behind it on the stream ``side``."""
        w, n = self.pack.struct, s.shape[0]
        ws = scratch.get(_nbytes("b200pf_single_track_rows_workspace", n, w.cs, w.hidden))
        call("b200pf_single_track_beside", ptr(s), ptr(z), C.byref(self.bias_struct), C.byref(w), ptr(bias), ptr(tok_mask_u8), n, ws, stream(), side,
             ready, done, int(wait_done))

    def finish(self, s_rows: torch.Tensor, og: torch.Tensor, scratch: Scratch) -> None:
        w = self.pack.struct
        ws = scratch.get(_nbytes("b200pf_single_track_workspace", s_rows.shape[0], w.cs, w.hidden))
        call("b200pf_single_track_finish", ptr(s_rows), C.byref(w), ptr(og), s_rows.shape[0], ws, stream())


class SingleTrackF32:
    """The same on the un-fused fp32 kernels: widths the part-plane kernels are not built for."""

    def __init__(self, sd, pre: str, num_heads: int, device) -> None:
        f32 = lambda name: weights.to_device_f32(sd, pre + name, device)
        self.num_heads = num_heads
        self.w_norm, self.w_att, self.w_trans = f32("pre_norm_s."), f32("attention."), f32("transition_s.")
        w_att, w_trans = self.w_att, self.w_trans
        cs = w_att["proj_q.weight"].shape[0]
        self.w_qg = torch.cat([w_att["proj_q.weight"], w_att["proj_g.weight"]], 0).contiguous()
        self.b_qg = torch.cat([w_att["proj_q.bias"], torch.zeros(cs, device=device)], 0).contiguous()
        self.w_kv = torch.cat([w_att["proj_k.weight"], w_att["proj_v.weight"]], 0).contiguous()
        self.w_12 = torch.cat([w_trans["fc1.weight"], w_trans["fc2.weight"]], 0).contiguous()

    def bias(self, z_rows: torch.Tensor) -> torch.Tensor:
        """bias[h][i_local * N + j]: one fp32 pass over the (local rows of) z [nr, N, c_z]."""
        w = self.w_att
        rows, c = z_rows.shape[0] * z_rows.shape[1], z_rows.shape[-1]
        heads = w["proj_z.1.weight"].shape[0]
        out = torch.empty(heads, rows, dtype=torch.float32, device=z_rows.device)
        if c == C_Z and heads in (4, 16):
            call("b200pf_ln_proj_heads", ptr(z_rows), ptr(w["proj_z.0.weight"]), ptr(w["proj_z.0.bias"]),
                 ptr(w["proj_z.1.weight"]), ptr(out), rows, rows, c, heads, stream())
        else:
            x = f32_layernorm(z_rows, w["proj_z.0.weight"], w["proj_z.0.bias"])
            call("b200pf_f32_linear_t", ptr(x), ptr(w["proj_z.1.weight"]), None, ptr(out), rows, rows, c, heads, stream())
        return out

    def attention(self, s: torch.Tensor, bias: torch.Tensor, tok_mask_u8: Optional[torch.Tensor], r0: int, nq: int, scratch: Scratch) -> torch.Tensor:
        n, cs = s.shape
        hd, st = cs // self.num_heads, stream()
        sn = f32_layernorm(s, self.w_norm["weight"], self.w_norm["bias"])
        qg = f32_linear(sn[r0:r0 + nq], self.w_qg, self.b_qg)                           # [nq, 2 cs]: q | g
        pitch = _round_up(n, 4)
        kvt = torch.empty(2 * cs, pitch, dtype=torch.float32, device=s.device)          # [k rows | v rows][key]
        call("b200pf_f32_linear_t", ptr(sn), ptr(self.w_kv), None, ptr(kvt), pitch, n, cs, 2 * cs, st)
        o = torch.empty(nq, cs, dtype=torch.float32, device=s.device)
        call("b200pf_f32_sattention", ptr(qg), 2 * cs, qg.data_ptr() + 4 * cs, 2 * cs, ptr(kvt), kvt.data_ptr() + 4 * cs * pitch, pitch,
             ptr(o), cs, ptr(bias), nq * n, n, ptr(tok_mask_u8), nq, n, self.num_heads, hd, 1.0 / math.sqrt(hd), 1e6, st)
        return o

    def rows(self, s: torch.Tensor, bias: torch.Tensor, tok_mask_u8: Optional[torch.Tensor], scratch: Scratch) -> None:
        self.finish(s, self.attention(s, bias, tok_mask_u8, 0, s.shape[0], scratch), scratch)

    def finish(self, s_rows: torch.Tensor, og: torch.Tensor, scratch: Scratch) -> None:
        n = s_rows.shape[0]
        f32_linear(og, self.w_att["proj_o.weight"], out=s_rows, accumulate=True)
        x = f32_layernorm(s_rows, self.w_trans["norm.weight"], self.w_trans["norm.bias"])
        h12 = f32_linear(x, self.w_12)                                                  # [n, 2 hidden]: fc1 | fc2
        hidden = h12.shape[1] // 2
        h = torch.empty(n, hidden, dtype=torch.float32, device=s_rows.device)
        call("b200pf_f32_gate_strided", ptr(h12), 2 * hidden, h12.data_ptr() + 4 * hidden, 2 * hidden, ptr(h), hidden,
             n, hidden, 1, stream())
        f32_linear(h, self.w_trans["fc3.weight"], out=s_rows, accumulate=True)


def single_track_fits(sd, pre: str, num_heads: int) -> bool:
    """Whether the part-plane kernels are built for the single track's widths: c_s = 384 (or 64, 128, 256), heads of 24 or 32, hidden
    a multiple of 64, a pair width and head count the bias projection is built for."""
    cs = sd[pre + "pre_norm_s.weight"].shape[0]
    hidden = sd[pre + "transition_s.fc1.weight"].shape[0]
    heads, cz = sd[pre + "attention.proj_z.1.weight"].shape
    return (cs in weights.SPLIT_WIDTHS + (384,) and cs % num_heads == 0 and cs // num_heads in (24, 32) and hidden % 64 == 0
            and cz in weights.SPLIT_WIDTHS and heads in (4, 8, 16))


def pack_single_track(sd, pre: str, num_heads: int, device, pack=None):
    """Part-plane kernels where their widths fit (``pack``: their weights where the caller has packed them), the un-fused fp32 kernels
    elsewhere."""
    if single_track_fits(sd, pre, num_heads):
        return SingleTrack(sd, pre, num_heads, device, pack)
    return SingleTrackF32(sd, pre, num_heads, device)


def single_track(s: torch.Tensor, z: torch.Tensor, tok_mask_u8: torch.Tensor, track, scratch: Scratch) -> None:
    """The single track of one layer on all rows."""
    track.rows(s, track.bias(z), tok_mask_u8, scratch)
