"""Python face of the atom-transformer layer's kernels (``csrc/atom_proj_sm100.cu``, ``csrc/window_layer_sm100.cu``): conditioned
norm -> q | k | v | gate projection, window attention with its output projection, conditioned transition.

They serve rows of 128 channels with 4 heads of 32; anything else takes the row kernels and the GEMM, one product at a time
(:mod:`ops.rows`, :mod:`ops.gemm`, :func:`ops.pair.window_attention_fused`).
"""
from __future__ import annotations

from typing import Optional

import torch

from . import gemm as _gemm
from . import native, pair, rows
from .native import c_int, c_ll, c_void_p

native.declare("ubm_atom_qkvg", [c_void_p] * 6 + [c_ll, c_ll, c_ll, c_void_p, c_void_p])
native.declare("ubm_window_layer", [c_void_p] * 6 + [c_int, c_int, c_int, c_ll, c_ll, c_void_p])
native.declare("ubm_cond_transition", [c_void_p] * 7 + [c_ll, c_ll, c_int, c_ll, c_ll, c_void_p, c_void_p])

C = 128


def _rows_of(t: Optional[torch.Tensor], R: int):
    """Conditioning rows as [rows, 128] whose 16-byte units the kernels can read in place (a column slice of a wider buffer is
    fine), or None.  A row serves every sample, so their number divides R."""
    if t is None or t.dtype != torch.bfloat16 or not t.is_cuda:
        return None
    t = rows._cond2d(t, C)
    if t.shape[0] == 0 or R % t.shape[0] or t.stride(0) % 8 or t.stride(0) < C or t.data_ptr() % 16:
        return None
    return t


def _gate_of(t: Optional[torch.Tensor], R: int):
    """The same for a gate, which is a matrix as it stands (the GEMM's epilogue takes no other)."""
    return _rows_of(t, R) if t is not None and t.dim() == 2 and t.shape[1] == C and t.stride(1) == 1 else None


def _plain(t: torch.Tensor) -> bool:
    return t.is_cuda and t.dtype == torch.bfloat16 and t.is_contiguous() and t.data_ptr() % 16 == 0


def _window_serves(w: pair.ApbPacked, bias: torch.Tensor, B: int, A: int, c: int) -> bool:
    return (pair.WINDOW_KERNEL == "tc" and c == C and w.wqkvg.shape == (4 * C, C) and w.H == 4 and w.Dp == 32 and
            w.wo.shape == (C, C) and A % 32 == 0 and A > 0
            and (bias is None or (_plain(bias) and bias.shape[0] in (1, B))))


def window_layer(qkvg: torch.Tensor, w: pair.ApbPacked, bias: Optional[torch.Tensor], gate: Optional[torch.Tensor],
                 residual: Optional[torch.Tensor], B: int, A: int) -> torch.Tensor:
    """residual + gate * proj_o(window attention) from qkvg [B * A, 512] (q scaled | k | v | sigmoid of the gate projection)."""
    out = torch.empty((B, A, C), dtype=torch.bfloat16, device=qkvg.device)
    rc = native.lib().ubm_window_layer(
        qkvg.data_ptr(), native.ptr(bias), w.wo.data_ptr(), native.ptr(gate), native.ptr(residual), out.data_ptr(), B, A,
        1 if bias is None else bias.shape[0], 0 if gate is None else gate.shape[0], 0 if gate is None else gate.stride(0),
        native.current_stream(qkvg.device))
    native.check(rc, "ubm_window_layer")
    return out


def attention(a: torch.Tensor, scale: torch.Tensor, shift: torch.Tensor, w: pair.ApbPacked, bias: torch.Tensor,
              gate: torch.Tensor) -> torch.Tensor:
    """a + gate * proj_o(window attention of sigmoid(scale) * LN(a) + shift).  a: bf16 [B, A, c], contiguous; gate: [rows, c], already
    a sigmoid; bias: :class:`models.diffusion.WindowBias` data."""
    B, A, c = a.shape
    R = B * A
    if c == C and _plain(a) and _window_serves(w, bias, B, A, c):
        sc, sh, gt = _rows_of(scale, R), _rows_of(shift, R), _gate_of(gate, R)
        if sc is not None and sh is not None and gt is not None and sc.shape == sh.shape and sc.stride(0) == sh.stride(0):
            qkvg = torch.empty((R, 4 * C), dtype=torch.bfloat16, device=a.device)
            rc = native.lib().ubm_atom_qkvg(a.data_ptr(), sc.data_ptr(), sh.data_ptr(), w.wqkvg.data_ptr(), w.bqkvg.data_ptr(),
                                            qkvg.data_ptr(), R, sc.shape[0], sc.stride(0),
                                            native.status_tensor(a.device).data_ptr(), native.current_stream(a.device))
            native.check(rc, "ubm_atom_qkvg")
            return window_layer(qkvg, w, bias, gt, a, B, A)
    return pair.window_attention_fused(rows.adaln_rows(a, scale, shift), w, bias, out_gate=gate, out_residual=a.view(R, c))


def transition(a: torch.Tensor, scale: torch.Tensor, shift: torch.Tensor, gate: torch.Tensor, w_in: torch.Tensor,
               w_out: torch.Tensor, packed: bool = True) -> torch.Tensor:
    """a + gate * (W_out (silu(g) * v * u)), g | v | u = W_in (sigmoid(scale) * LN(a) + shift).  ``packed``: the rows of W_in come as
    :func:`ops.gemm.pack_swiglu3` lays them out."""
    B, A, c = a.shape
    R = B * A
    if c == C and packed and _plain(a) and w_out.shape[0] == C and w_in.shape == (3 * w_out.shape[1], C):
        sc, sh, gt = _rows_of(scale, R), _rows_of(shift, R), _gate_of(gate, R)
        if (sc is not None and sh is not None and gt is not None and sc.shape == sh.shape == gt.shape
                and sc.stride(0) == sh.stride(0) and sc.shape[0] >= 128):
            # tiles of 128 rows do not cross from one run of conditioning rows to the next: runs shorter than a tile waste it
            out = torch.empty_like(a)
            rc = native.lib().ubm_cond_transition(
                a.data_ptr(), sc.data_ptr(), sh.data_ptr(), gt.data_ptr(), w_in.data_ptr(), w_out.data_ptr(), out.data_ptr(), R,
                sc.shape[0], w_out.shape[1], sc.stride(0), gt.stride(0), native.status_tensor(a.device).data_ptr(),
                native.current_stream(a.device))
            native.check(rc, "ubm_cond_transition")
            return out
    x = rows.adaln_rows(a, scale, shift).view(R, c)
    u = _gemm.gemm(x, w_in, act="swiglu3") if packed else rows.swiglu3_rows(_gemm.gemm(x, w_in))
    return _gemm.gemm(u, w_out, gate=gate, residual=a.view(R, c)).view(B, A, c)
