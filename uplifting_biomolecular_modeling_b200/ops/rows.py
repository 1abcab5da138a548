"""Python face of the row kernels (``csrc/rows_sm100.cu``): LayerNorm rows, pair -> head-bias
planes, AdaLN, gated residual, SwiGLU.  Each wrapper has the same signature as its plain
statement in :mod:`ops.reference` where one exists."""
from __future__ import annotations

import weakref
from typing import Optional

import torch

from . import native
from .native import c_float, c_int, c_ll, c_void_p

native.declare("ubm_layernorm_rows", [c_void_p] * 4 + [c_ll, c_int, c_float, c_int, c_int, c_void_p])
native.declare("ubm_outer_proj", [c_void_p] * 7 + [c_ll, c_float, c_void_p])
native.declare("ubm_pair_head_bias", [c_void_p] * 5 + [c_int, c_int, c_int, c_int, c_void_p])
native.declare("ubm_adaln_rows", [c_void_p] * 4 + [c_ll, c_int, c_ll, c_ll, c_float, c_void_p])
native.declare("ubm_gate_residual", [c_void_p] * 4 + [c_ll, c_int, c_ll, c_ll, c_void_p])
native.declare("ubm_swiglu_rows", [c_void_p] * 2 + [c_ll, c_int, c_void_p])
native.declare("ubm_swiglu3_rows", [c_void_p] * 2 + [c_ll, c_int, c_void_p])
native.declare("ubm_segment_mean", [c_void_p] * 3 + [c_int] * 5 + [c_void_p])
native.declare("ubm_gather_rows_add", [c_void_p] * 4 + [c_int] * 4 + [c_void_p])
native.declare("ubm_mean_rescale", [c_void_p] * 3 + [c_ll, c_int, c_float, c_void_p])

_DT = {torch.bfloat16: 0, torch.float32: 1}


_F32_CACHE: dict = {}


def _f32_param(t: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    """Contiguous fp32 copy of an affine parameter, kept until the parameter is written again (the conversion was two
    small launches per LayerNorm call)."""
    if t is None:
        return None
    if t.dtype == torch.float32 and t.is_contiguous():
        return t
    ent = _F32_CACHE.get(id(t))
    if ent is None or ent[0] is not t or ent[1] != t._version or ent[2].device != t.device:
        if len(_F32_CACHE) > 4096:
            _F32_CACHE.clear()
        ent = (t, t._version, t.detach().float().contiguous())
        _F32_CACHE[id(t)] = ent
    return ent[2]


def layernorm_rows(x: torch.Tensor, weight: Optional[torch.Tensor], bias: Optional[torch.Tensor],
                   eps: float = 1e-5, out_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    if x.dtype not in _DT or not x.is_contiguous():
        raise ValueError("layernorm_rows expects contiguous bf16 / fp32 input")
    C = x.shape[-1]
    R = x.numel() // C
    out_dtype = out_dtype or x.dtype
    out = torch.empty(x.shape, dtype=out_dtype, device=x.device)
    w, b = _f32_param(weight), _f32_param(bias)
    rc = native.lib().ubm_layernorm_rows(native.ptr(x), native.ptr(w), native.ptr(b), native.ptr(out), R, C,
                                         float(eps), _DT[x.dtype], _DT[out_dtype], native.current_stream(x.device))
    native.check(rc, "ubm_layernorm_rows")
    return out


def mean_rescale_(o: torch.Tensor, count: torch.Tensor, bias: torch.Tensor, total: float) -> torch.Tensor:
    """o[r] = o[r] * total / max(count[r], 1) + bias in place.  o: bf16 [R, C], contiguous; count: R fp32 elements;
    bias: fp32 [C]."""
    R, C = o.shape
    if o.dtype != torch.bfloat16 or not o.is_contiguous() or count.dtype != torch.float32 or count.numel() != R or \
            not count.is_contiguous() or bias.dtype != torch.float32 or bias.shape != (C,) or not bias.is_contiguous():
        raise ValueError(f"mean_rescale_ expects bf16 rows with {R} fp32 counts and {C} fp32 biases")
    if not o.is_cuda or count.device != o.device or bias.device != o.device:
        raise ValueError("mean_rescale_: rows, counts and biases live on one GPU")
    if bias.data_ptr() % 16:                                    # read four at a time
        bias = bias.clone()
    rc = native.lib().ubm_mean_rescale(native.ptr(o), native.ptr(count), native.ptr(bias), R, C, float(total),
                                       native.current_stream(o.device))
    native.check(rc, "ubm_mean_rescale")
    return o


_HB_CACHE: dict = {}


def _kept(t: Optional[torch.Tensor]) -> tuple:
    """What tells later whether ``t`` is still the tensor, with the contents, that something was made from: the object (weakly), its
    version, and its storage, held so that no other can have its address (a converted copy swaps ``.data`` and leaves the version)."""
    return (lambda: None, 0, 0, None) if t is None else (weakref.ref(t), t._version, t.data_ptr(), t.detach())


def _unchanged(kept: tuple, t: Optional[torch.Tensor]) -> bool:
    return kept[0]() is t and (t is None or (kept[1] == t._version and kept[2] == t.data_ptr()))


def _head_bias_weights(w: torch.Tensor, ln_w, ln_b, scale: float, device) -> tuple:
    """(fp32 weights with the norm's scale folded in, their row sums, their products with the norm's shift), kept until the weight or
    either parameter of the norm is another one or is written."""
    key = (id(w), scale, device)
    entry = _HB_CACHE.get(key)
    if entry is not None and _unchanged(entry[0], w) and _unchanged(entry[1], ln_w) and _unchanged(entry[2], ln_b):
        return entry[3]
    gam = torch.ones(128, device=device) if ln_w is None else ln_w.detach().float()
    wf = (w.detach().float() * gam[None, :] * scale).contiguous()
    colsum = wf.sum(1).contiguous()
    colbias = torch.zeros(w.shape[0], device=device) if ln_b is None else \
        ((w.detach().float() @ ln_b.detach().float()) * scale).contiguous()
    if len(_HB_CACHE) > 4096:
        _HB_CACHE.clear()
    _HB_CACHE[key] = (_kept(w), _kept(ln_w), _kept(ln_b), (wf, colsum, colbias))
    return wf, colsum, colbias


def pair_head_bias(z: torch.Tensor, ln_w, ln_b, w, scale: float = 1.0, transpose: bool = False,
                   out: Optional[torch.Tensor] = None, row: int = 16) -> torch.Tensor:
    """z: bf16 [N, N, 128]; w: [H, 128].  Returns bf16 [H, N, N] (a view of planes whose rows are padded with zeros to a
    multiple of ``row`` elements, 8 or more) with ``scale * Linear(LN(z))`` laid out head-major.  ``out``: bf16 planes [H, N, N or more] to
    write instead, one behind the other with rows of a multiple of 8 elements; columns behind N are left as they are."""
    N = z.shape[0]
    H = w.shape[0]
    # Whole 32-byte sectors (16): the contraction of the pair-weighted averaging reads the planes and values of their row length
    # (760 tokens x 1024 sequences 845 -> 701 us, 405 x 500 221 -> 204).  The attention's bias tiles gain nothing (602 us both ways),
    # and where only they are padded (136 tokens) the fill costs 1 us of 4.8: it asks for 8.
    if out is not None:
        Np = out.stride(1) if out.dim() == 3 else 0
        if out.dtype != torch.bfloat16 or out.device != z.device or out.dim() != 3 or out.shape[0] < H or out.shape[1] != N or \
                out.shape[2] < N or out.stride(2) != 1 or Np < N or Np % 8 or out.stride(0) != N * Np:
            raise ValueError(f"pair_head_bias: planes of {H} heads are bf16 [{H}, {N}, {N} or more], rows of a multiple of 8 elements")
    else:
        if row < 8 or row % 8:
            raise ValueError("pair_head_bias: rows of a multiple of 8 elements")
        Np = (N + row - 1) // row * row
        make = torch.zeros if Np != N else torch.empty       # the kernel writes no padding
        out = make((H, N, Np), dtype=torch.bfloat16, device=z.device)
    wf, colsum, colbias = _head_bias_weights(w, ln_w, ln_b, scale, z.device)
    rc = native.lib().ubm_pair_head_bias(native.ptr(z), native.ptr(wf), native.ptr(colsum), native.ptr(colbias),
                                         native.ptr(out), N, Np, H, 1 if transpose else 0,
                                         native.current_stream(z.device))
    native.check(rc, "ubm_pair_head_bias")
    return out[:, :, :N]


def outer_projections(m: torch.Tensor, ln_w, ln_b, eps: float, wa: torch.Tensor, wb: torch.Tensor,
                      mask: Optional[torch.Tensor]) -> torch.Tensor:
    """bf16 [2, R, 32]: the projections by wa and wb (bf16 [32, 64]) of LN(m), times the row's mask.  m: bf16 [R, 64], contiguous, on 16
    bytes; mask: bf16 [R], contiguous, or None."""
    R = m.shape[0]
    if m.dtype != torch.bfloat16 or m.shape != (R, 64) or not m.is_contiguous() or wa.shape != (32, 64) or wb.shape != (32, 64) or \
            wa.dtype != torch.bfloat16 or wb.dtype != torch.bfloat16 or wa.device != m.device or wb.device != m.device or \
            (mask is not None and (mask.dtype != torch.bfloat16 or mask.shape != (R,) or not mask.is_contiguous() or
                                   mask.device != m.device)):
        raise ValueError("outer_projections: bf16 rows of 64 channels, two weights of [32, 64], a mask of one value per row")
    out = torch.empty((2, R, 32), dtype=torch.bfloat16, device=m.device)
    wa, wb, g, b = wa.contiguous(), wb.contiguous(), _f32_param(ln_w), _f32_param(ln_b)
    rc = native.lib().ubm_outer_proj(native.ptr(m), native.ptr(g), native.ptr(b), native.ptr(wa), native.ptr(wb), native.ptr(mask),
                                     native.ptr(out), R, float(eps), native.current_stream(m.device))
    native.check(rc, "ubm_outer_proj")
    return out


def _cond2d(t: torch.Tensor, C: int) -> torch.Tensor:
    """Conditioning rows as a 2-D view [rows, C] whose rows may be strided (a column slice of a wider buffer)."""
    t2 = t.reshape(-1, C) if t.is_contiguous() else t.squeeze(0) if t.dim() == 3 and t.shape[0] == 1 else t
    if t2.dim() != 2 or t2.shape[1] != C or t2.stride(1) != 1:
        t2 = t.reshape(-1, C).contiguous()
    return t2


def adaln_rows(a: torch.Tensor, scale: torch.Tensor, shift: torch.Tensor, eps: float = 1e-5) -> torch.Tensor:
    """sigmoid(scale) * LN_noaffine(a) + shift; scale/shift rows are reused cyclically over a's rows and may be
    column slices of one wider buffer (equal row strides)."""
    C = a.shape[-1]
    R = a.numel() // C
    out = torch.empty_like(a)
    sc, sh = _cond2d(scale, C), _cond2d(shift, C)
    if sc.stride(0) != sh.stride(0) or sc.shape[0] != sh.shape[0]:
        sc, sh = sc.contiguous(), sh.contiguous()
    rc = native.lib().ubm_adaln_rows(native.ptr(a), native.ptr(sc), native.ptr(sh), native.ptr(out), R, C,
                                     sc.shape[0], sc.stride(0), float(eps), native.current_stream(a.device))
    native.check(rc, "ubm_adaln_rows")
    return out


def gate_residual(x: torch.Tensor, gate: torch.Tensor, res: Optional[torch.Tensor]) -> torch.Tensor:
    """res + sigmoid(gate) * x; gate rows reused cyclically, possibly a column slice of a wider buffer."""
    C = x.shape[-1]
    R = x.numel() // C
    out = torch.empty_like(x)
    g = _cond2d(gate, C)
    rc = native.lib().ubm_gate_residual(native.ptr(x), native.ptr(g), native.ptr(res), native.ptr(out), R, C,
                                        g.shape[0], g.stride(0), native.current_stream(x.device))
    native.check(rc, "ubm_gate_residual")
    return out


def swiglu3_rows(x: torch.Tensor) -> torch.Tensor:
    """x: [.., 3*Hd] = [u | g | w] -> silu(u) * g * w."""
    Hd = x.shape[-1] // 3
    R = x.numel() // (3 * Hd)
    out = torch.empty(x.shape[:-1] + (Hd,), dtype=x.dtype, device=x.device)
    rc = native.lib().ubm_swiglu3_rows(native.ptr(x), native.ptr(out), R, Hd, native.current_stream(x.device))
    native.check(rc, "ubm_swiglu3_rows")
    return out


def swiglu_rows(ab: torch.Tensor) -> torch.Tensor:
    Hd = ab.shape[-1] // 2
    R = ab.numel() // (2 * Hd)
    out = torch.empty(ab.shape[:-1] + (Hd,), dtype=ab.dtype, device=ab.device)
    rc = native.lib().ubm_swiglu_rows(native.ptr(ab), native.ptr(out), R, Hd, native.current_stream(ab.device))
    native.check(rc, "ubm_swiglu_rows")
    return out


def segment_mean(t: torch.Tensor, table: torch.Tensor, n_tokens: int) -> torch.Tensor:
    """Mean of atom rows per token.  t: bf16 [B, A, C]; table: int32 [N, M] atom indices (-1 = none)."""
    t = t.contiguous()
    B, A, C = t.shape
    out = torch.empty((B, n_tokens, C), dtype=t.dtype, device=t.device)
    rc = native.lib().ubm_segment_mean(native.ptr(t), native.ptr(table), native.ptr(out), B, A, n_tokens,
                                       table.shape[1], C, native.current_stream(t.device))
    native.check(rc, "ubm_segment_mean")
    return out


def gather_rows_add(q: Optional[torch.Tensor], a: torch.Tensor, a2t: torch.Tensor) -> torch.Tensor:
    """q + a[:, a2t] (token rows broadcast to their atoms).  q: bf16 [B, A, C] or None; a: [B, N, C]; a2t: int32 [A]."""
    a = a.contiguous()
    B, N, C = a.shape
    A = a2t.shape[0]
    out = torch.empty((B, A, C), dtype=a.dtype, device=a.device)
    qq = None if q is None else q.contiguous()
    rc = native.lib().ubm_gather_rows_add(native.ptr(qq), native.ptr(a), native.ptr(a2t), native.ptr(out), B, A, N, C,
                                          native.current_stream(a.device))
    native.check(rc, "ubm_gather_rows_add")
    return out
