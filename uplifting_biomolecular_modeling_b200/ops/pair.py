"""Python face of the fused pair-stack kernels (triangle multiplication, pair transition,
triangle attention).  Weight preparation ("folding") happens once per module:

* LayerNorm is folded into the following Linear: ``W' = W * gamma`` (bf16), with the per-column
  constants ``colsum = rowsum(W')`` and ``colbias = W @ beta (+ bias)`` in fp32, so that
  ``Linear(LN(x)) = rstd * (W' x - mu * colsum) + colbias`` and the kernels feed raw rows to the
  tensor cores.
* Matrices that the kernels consume side by side are stacked in the order the kernel expects.

The reference performs the same kind of one-time weight work in its "castcache"/"interleave fold"
levers (common/opt_core/opt_core/of3_trunk/castcache.py, evo2/CHANGES.md lever L2).
"""
from __future__ import annotations

import ctypes
import struct
from dataclasses import dataclass
from typing import Optional

import torch
import torch.nn.functional as F

from . import gemm as _gemm
from . import native
from .native import c_float, c_int, c_ll, c_void_p

native.declare("ubm_trimul_proj", [c_void_p] * 7 + [c_int, c_int, c_void_p, c_void_p])
native.declare("ubm_triatt_proj", [c_void_p] * 13 + [c_int, c_int, c_int, c_int, c_void_p, c_void_p])
native.declare("ubm_trimul_out", [c_void_p] * 9 + [c_int, c_int, c_int, c_void_p, c_void_p])
native.declare("ubm_transition", [c_void_p] * 8 + [c_ll, c_int, c_int, c_void_p, c_void_p])
# row-block forms (also the per-rank forms of the row-sharded pair stack)
native.declare("ubm_trimul_proj_rows", [c_void_p] * 7 + [c_int, c_int, c_int, c_int, c_void_p, c_void_p])
native.declare("ubm_triatt_proj_rows", [c_void_p] * 13 + [c_int, c_int, c_int, c_int, c_int, c_int, c_void_p, c_void_p])
native.declare("ubm_trimul_out_rows", [c_void_p] * 9 + [c_int, c_int, c_int, c_int, c_void_p, c_void_p])


# whole operators from one call (csrc/sequences_sm100.cu): their arguments as 8-byte integers, in the order the library reads them
for _name in ("ubm_trimul", "ubm_triatt", "ubm_pair_track", "ubm_single_track", "ubm_apb", "ubm_transition_rows"):
    native.declare(_name, [ctypes.c_char_p])
_TRIMUL_ARGS, _TRIATT_ARGS, _APB_ARGS = struct.Struct("=21q"), struct.Struct("=26q"), struct.Struct("=28q")
_TRANSITION_ROWS_ARGS, _PAIR_TRACK_ARGS, _SINGLE_TRACK_ARGS = struct.Struct("=3qd12q"), struct.Struct("=56q"), struct.Struct("=14q2d23q")


def ceil_to(n: int, m: int) -> int:
    return (n + m - 1) // m * m


def fold_ln_linear(W: torch.Tensor, gamma: Optional[torch.Tensor], beta: Optional[torch.Tensor],
                   bias: Optional[torch.Tensor] = None, scale: float = 1.0):
    """Returns (W' bf16 [out, in], colsum fp32 [out], colbias fp32 [out]) for Linear(LN(x)) * scale."""
    Wf = W.detach().float()
    g = torch.ones(Wf.shape[1], device=Wf.device) if gamma is None else gamma.detach().float()
    Wg = (Wf * g[None, :]) * scale
    Wb = Wg.to(torch.bfloat16).contiguous()
    colsum = Wb.float().sum(dim=1).contiguous()
    colbias = torch.zeros(Wf.shape[0], device=Wf.device)
    if beta is not None:
        colbias = colbias + Wf @ beta.detach().float()
    if bias is not None:
        colbias = colbias + bias.detach().float()
    return Wb, colsum, (colbias * scale).contiguous()


# ------------------------------------------------------------------------------------------
@dataclass
class TransitionPacked:
    wab: torch.Tensor       # bf16 [(hidden/64)*128, 128]
    wo: torch.Tensor        # bf16 [128, hidden]
    colsum: torch.Tensor    # fp32 [(hidden/64)*128]
    colbias: torch.Tensor
    hidden: int

    @classmethod
    def pack(cls, norm_w, norm_b, fc1, fc2, fc3) -> "TransitionPacked":
        hidden, c = fc1.shape
        if c != 128 or hidden % 64 or hidden > 1024:
            raise ValueError(f"fused transition supports c=128 and hidden%64==0, <=1024 (got c={c}, hidden={hidden})")
        a, a_sum, a_bias = fold_ln_linear(fc1, norm_w, norm_b)
        b, b_sum, b_bias = fold_ln_linear(fc2, norm_w, norm_b)
        wo = fc3.detach().to(torch.bfloat16).contiguous()
        if hidden == 64:
            # the kernel's pipeline runs two chunks ahead of its output and takes two chunks of 64 or more; a chunk of
            # zero weights adds silu(0) * 0 = 0
            hidden = 128
            a, b = F.pad(a, (0, 0, 0, 64)), F.pad(b, (0, 0, 0, 64))
            a_sum, b_sum, a_bias, b_bias = (F.pad(t, (0, 64)) for t in (a_sum, b_sum, a_bias, b_bias))
            wo = F.pad(wo, (0, 64))
        nch = hidden // 64
        wab = torch.stack([a.view(nch, 64, c), b.view(nch, 64, c)], dim=1).reshape(nch * 128, c).contiguous()
        colsum = torch.stack([a_sum.view(nch, 64), b_sum.view(nch, 64)], dim=1).reshape(-1).contiguous()
        colbias = torch.stack([a_bias.view(nch, 64), b_bias.view(nch, 64)], dim=1).reshape(-1).contiguous()
        return cls(wab, wo, colsum, colbias, hidden)


def _result(out: Optional[torch.Tensor], like: torch.Tensor, rows_apart: bool = False) -> torch.Tensor:
    """A new result in the form of ``like``, or the caller's ``out``: the kernels write it by its address alone, so it has to be bf16 on
    the same GPU with its elements side by side; with ``rows_apart`` (its rows are addressed block by block) of the same shape, too."""
    if out is None:
        return torch.empty_like(like)
    if out.dtype != torch.bfloat16 or out.device != like.device or not out.is_contiguous() or out.numel() != like.numel() or \
            (rows_apart and out.shape != like.shape):
        raise ValueError(f"output of shape {tuple(out.shape)} ({out.dtype}, {out.device}) does not hold a contiguous bf16 result of shape "
                         f"{tuple(like.shape)} on {like.device}")
    return out


def transition_fused(x: torch.Tensor, w: TransitionPacked, residual: bool = True,
                     out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """x: bf16 [..., 128] contiguous.  Returns x + transition(x) (or the update alone)."""
    if x.dtype != torch.bfloat16 or x.shape[-1] != 128 or not x.is_contiguous():
        raise ValueError("transition_fused expects a contiguous bf16 tensor with 128 channels")
    R = x.numel() // 128
    out = _result(out, x)
    st = native.status_tensor(x.device)
    rc = native.lib().ubm_transition(native.ptr(x), native.ptr(w.wab), native.ptr(w.wo), native.ptr(w.colsum),
                                     native.ptr(w.colbias), 0, 0, native.ptr(out), R, w.hidden,
                                     1 if residual else 0, native.ptr(st), native.current_stream(x.device))
    native.check(rc, "ubm_transition")
    return out


def transition_rows(x: torch.Tensor, norm_w, norm_b, eps: float, w12: torch.Tensor, w3: torch.Tensor, residual: bool) -> torch.Tensor:
    """Transition of other widths in one call: x bf16 [R, dim] contiguous, w12 as ``gemm.pack_swiglu`` packs it, w3 bf16 [out, hidden]."""
    from . import rows as _rows
    R, dim = x.shape
    out_dim, hidden = w3.shape
    if w12.shape != (2 * hidden, dim) or (residual and out_dim != dim) or x.dtype != torch.bfloat16 or w12.dtype != torch.bfloat16 or \
            w3.dtype != torch.bfloat16 or not x.is_contiguous() or not w12.is_contiguous() or not w3.is_contiguous():
        raise ValueError(f"transition_rows: contiguous bf16 rows and weights, {tuple(w12.shape)} and {tuple(w3.shape)} for {tuple(x.shape)}")
    dev = x.device
    g, b = _rows._f32_param(norm_w), _rows._f32_param(norm_b)
    scratch = torch.empty(R * (dim + hidden), dtype=torch.bfloat16, device=dev)      # norm rows, then hidden rows
    n = scratch.data_ptr()
    out = torch.empty((R, out_dim), dtype=torch.bfloat16, device=dev)
    rc = native.lib().ubm_transition_rows(_TRANSITION_ROWS_ARGS.pack(
        x.data_ptr(), native.ptr(g), native.ptr(b), eps, w12.data_ptr(), w3.data_ptr(), x.data_ptr() if residual else 0,
        n, n + 2 * R * dim, out.data_ptr(), R, dim, hidden, out_dim, native.status_tensor(dev).data_ptr(),
        native.current_stream(dev)))
    native.check(rc, "ubm_transition_rows")
    return out


# ------------------------------------------------------------------------------------------
@dataclass
class TrimulPacked:
    w_in: torch.Tensor       # bf16 [512, 128] rows [p_a; g_a; p_b; g_b]
    in_colsum: torch.Tensor  # fp32 [512]
    in_colbias: torch.Tensor
    wo: torch.Tensor         # bf16 [128, 128]
    o_colsum: torch.Tensor
    o_colbias: torch.Tensor
    wg: torch.Tensor         # bf16 [128, 128]
    g_colsum: torch.Tensor
    g_colbias: torch.Tensor

    @classmethod
    def pack(cls, norm_in_w, norm_in_b, p_in, g_in, norm_out_w, norm_out_b, p_out, g_out) -> "TrimulPacked":
        two_h, c = p_in.shape
        if c != 128 or two_h != 256:
            raise ValueError("fused triangle multiplication supports c_z = c_hidden = 128")
        h = two_h // 2
        stacked = torch.cat([p_in[:h], g_in[:h], p_in[h:], g_in[h:]], dim=0)
        w_in, s_in, b_in = fold_ln_linear(stacked, norm_in_w, norm_in_b)
        wo, so, bo = fold_ln_linear(p_out, norm_out_w, norm_out_b)
        wg, sg, bg = fold_ln_linear(g_out, norm_in_w, norm_in_b)
        return cls(w_in, s_in, b_in, wo, so, bo, wg, sg, bg)

    def pointers(self) -> tuple:
        return (self.w_in.data_ptr(), self.in_colsum.data_ptr(), self.in_colbias.data_ptr(), self.wo.data_ptr(),
                self.o_colsum.data_ptr(), self.o_colbias.data_ptr(), self.wg.data_ptr(), self.g_colsum.data_ptr(),
                self.g_colbias.data_ptr())


# Elements by which a row of the channel-major planes is padded: whole 32-byte sectors.  On 16 bytes (8 elements), which is all
# that TMA asks for, every box of every other row begins and ends inside a sector, and projection, contraction and output stage
# write those in parts: 1818 -> 1575 us (outgoing), 1945 -> 1693 (incoming) at 1400 tokens, 134 -> 126 and 132 -> 126 at 401,
# 427 -> 420 and 504 -> 502 at 777.  Whole lines (64 elements) add nothing and cost their bytes (650 incoming: 285 -> 304).
PLANE_ROW = 16


def _trimul_blocked(z, m, w: TrimulPacked, outgoing: bool, residual: bool, out, ws: dict, rb: int):
    """Row-blocked triangle multiplication: the projected operand planes a, b exist whole (the contraction of a
    row block needs every row of the other operand), the contracted planes x only for ``rb`` rows of the update
    at a time - contraction and output stage alternate per block.  Same kernels, same sums as the whole form."""
    N = z.shape[0]
    Np = ceil_to(N, PLANE_ROW)
    dev = z.device
    out = _result(out, z, rows_apart=True)
    key = ("trimul_blocked", N, rb, dev)
    if key not in ws:
        ws[key] = (torch.empty((2, 128, N, Np), dtype=torch.bfloat16, device=dev),
                   torch.empty((128, rb, Np), dtype=torch.bfloat16, device=dev))
    planes, xb = ws[key]
    st = native.status_tensor(dev)
    stream = native.current_stream(dev)
    lib = native.lib()
    rc = lib.ubm_trimul_proj(native.ptr(z), native.ptr(w.w_in), native.ptr(w.in_colsum), native.ptr(w.in_colbias),
                             native.ptr(m), native.ptr(planes), 0, N, Np, native.ptr(st), stream)
    native.check(rc, "ubm_trimul_proj")
    for r0 in range(0, N, rb):
        r1 = min(N, r0 + rb)
        xv = xb.view(-1)[: 128 * (r1 - r0) * Np].view(128, r1 - r0, Np)
        if outgoing:      # x[c, i, j] = sum_k a[c, i, k] b[c, j, k]: rows i of a against all of b
            _gemm.gemm(planes[0][:, r0:r1, :N], planes[1][:, :, :N], out=xv[:, :, :N])
        else:             # x[c, i, j] = sum_k a[c, k, i] b[c, k, j]: columns i of a (MN-major operands)
            _gemm.gemm(planes[0][:, :, r0:r1], planes[1][:, :, :N], mn_major=True, out=xv[:, :, :N])
        rc = lib.ubm_trimul_out_rows(native.ptr(xv), native.ptr(z[r0:r1]), native.ptr(w.wo), native.ptr(w.wg),
                                     native.ptr(w.o_colsum), native.ptr(w.o_colbias), native.ptr(w.g_colsum),
                                     native.ptr(w.g_colbias), native.ptr(out[r0:r1]), r1 - r0, N, Np,
                                     1 if residual else 0, native.ptr(st), stream)
        native.check(rc, "ubm_trimul_out_rows")
    return out


def _trimul_scratch(ws: dict, N: int, Np: int, dev) -> tuple:
    key = ("trimul", N, dev)
    if key not in ws:
        ws[key] = (torch.empty((2, 128, N, Np), dtype=torch.bfloat16, device=dev),
                   torch.empty((128, N, Np), dtype=torch.bfloat16, device=dev))
    return ws[key]


def trimul_fused(z: torch.Tensor, mask: Optional[torch.Tensor], w: TrimulPacked, outgoing: bool,
                 residual: bool = True, out: Optional[torch.Tensor] = None,
                 workspace: Optional[dict] = None) -> torch.Tensor:
    """z: bf16 [N, N, 128] contiguous; mask: [N, N], sizes of one broadcast to it, or None.  Three launches: projection ->
    batched tcgen05 contraction -> output stage.  With ``workspace["row_block"]`` set (the ``chunk_pair_ops`` lever)
    and smaller than N, contraction and output stage run per block of rows (see :func:`_trimul_blocked`)."""
    if z.dtype != torch.bfloat16 or z.dim() != 3 or z.shape[-1] != 128 or not z.is_contiguous():
        raise ValueError("trimul_fused expects a contiguous bf16 [N, N, 128] tensor")
    N = z.shape[0]
    Np = ceil_to(N, PLANE_ROW)
    dev = z.device
    ws = workspace if workspace is not None else {}
    rb = int(ws.get("row_block", 0) or 0)
    if mask is not None and mask.shape != (N, N):
        # the kernel reads N * N values in this order; one row or column stands for all
        mask = mask.reshape(N, N) if mask.numel() == N * N else mask.expand(N, N)
    if 0 < rb < N:
        m = None if mask is None else mask.to(dev, torch.float32).contiguous()
        return _trimul_blocked(z, m, w, outgoing, residual, out, ws, rb // 8 * 8 or 8)
    out = _result(out, z)
    planes, x = _trimul_scratch(ws, N, Np, dev)
    kind = 0
    if mask is not None:
        # a bf16 mask of the pair tensor is read as it is; others are converted
        kind = 2 if mask.dtype == torch.bfloat16 and mask.shape == (N, N) and mask.device == dev and mask.is_contiguous() else 1
        if kind == 1:
            mask = mask.to(dev, torch.float32).contiguous()
    rc = native.lib().ubm_trimul(_TRIMUL_ARGS.pack(
        z.data_ptr(), 0 if mask is None else mask.data_ptr(), kind, *w.pointers(), planes.data_ptr(), x.data_ptr(), out.data_ptr(), N, Np,
        1 if outgoing else 0, 1 if residual else 0, native.status_tensor(dev).data_ptr(), native.current_stream(dev)))
    native.check(rc, "ubm_trimul")
    return out


# ------------------------------------------------------------------------------------------
_ATTN_SIG = [c_void_p] * 8 + [c_int, c_int, c_int, c_int, c_ll, c_ll, c_ll, c_ll, c_int, c_void_p, c_void_p]
native.declare("ubm_attention_d32", _ATTN_SIG)
native.declare("ubm_attention_d64", _ATTN_SIG)

native.declare("ubm_attention_set_variant", [c_int])
native.declare("ubm_key_mask", [c_void_p, c_int, c_ll, c_ll, c_void_p, c_void_p, c_int, c_int, c_void_p])

LOG2E = 1.4426950408889634


def set_attention_variant(v: int) -> None:
    """Low nibble, head dimension 32: 0 = choose by row count (four rows per CTA from four rows on), 5 = two rows
    with 128-key steps, 1 = two rows, P and bias through shared memory.  Bits 4-5: 0 = one exponential in four as a
    polynomial on the FMA pipe, 1 = all on the special-function unit."""
    native.lib().ubm_attention_set_variant(int(v))


MASK_STEP = 64          # the kernel's flags are per 64-key step
MASK_NEG = -1.0e30


@dataclass
class KeyMask:
    """A key mask laid out for the attention kernel: additive bf16 rows (0 keeps, -1e30 masks) padded to whole
    64-key steps, and one flag byte per (row, step) that is set when the step holds a masked key, so that rows and
    steps without masked keys run the mask-free loop (the reference skips the mask the same way for unmasked row
    groups: common/opt_core/opt_core/kernels/flash_triattn.py:35-37)."""
    add: torch.Tensor        # bf16 [rows, ld]
    flags: torch.Tensor      # uint8 [rows, ld / 64]

    @classmethod
    def pack(cls, keep: torch.Tensor) -> Optional["KeyMask"]:
        """keep: [rows, Nk], non-zero = attend.  Returns None when nothing is masked (one host read)."""
        keep = keep != 0
        if bool(keep.all()):
            return None
        rows, nk = keep.shape
        ld = ceil_to(nk, MASK_STEP)
        add = torch.zeros((rows, ld), dtype=torch.bfloat16, device=keep.device)
        add[:, :nk].masked_fill_(~keep, MASK_NEG)
        flags = (add.view(rows, ld // MASK_STEP, MASK_STEP) != 0).any(-1).to(torch.uint8).contiguous()
        return cls(add, flags)

    @classmethod
    def lay_out(cls, keep: torch.Tensor, shape: Optional[tuple] = None,
                device: Optional[torch.device] = None) -> "KeyMask":
        """:meth:`pack` of a mask as one launch and without the host read: a mask that keeps everything gets clear
        flags, with which the kernel runs its mask-free loop.  ``shape`` = (rows, Nk) that sizes of one broadcast to, ``device`` = the
        GPU it is wanted on (a mask made on the host is copied there)."""
        keep = cls.readable(keep, shape, device)
        rows, nk = keep.shape
        steps = ceil_to(nk, MASK_STEP) // MASK_STEP
        add = torch.empty((rows, steps * MASK_STEP), dtype=torch.bfloat16, device=keep.device)
        flags = torch.empty((rows, steps), dtype=torch.uint8, device=keep.device)
        rc = native.lib().ubm_key_mask(native.ptr(keep), keep.element_size(), keep.stride(0), keep.stride(1),
                                       native.ptr(add), native.ptr(flags), rows, nk, native.current_stream(keep.device))
        native.check(rc, "ubm_key_mask")
        return cls(add, flags)


    @staticmethod
    def readable(keep: torch.Tensor, shape: Optional[tuple], device: Optional[torch.device]) -> torch.Tensor:
        """The mask as the laying-out kernel reads it: on the GPU, of its full size (strides free), a type of 1, 2 or 4 bytes."""
        if device is not None and keep.device != device:
            keep = keep.to(device)
        if not keep.is_cuda:
            raise ValueError("a key mask is laid out on a GPU")
        if shape is not None and 1 in keep.shape:
            keep = keep.expand(*(to if n == 1 else -1 for n, to in zip(keep.shape, shape)))
        if keep.dtype not in (torch.float32, torch.bfloat16, torch.bool, torch.uint8):
            keep = keep != 0
        return keep


@dataclass
class TriattPacked:
    w: torch.Tensor          # bf16 [512, 128] rows [q * log2e/sqrt(d); k; v; g], gamma folded
    colsum: torch.Tensor     # fp32 [512]
    colbias: torch.Tensor
    wb: torch.Tensor         # fp32 [H, 128] head-bias weights * gamma * log2e
    wb_colsum: torch.Tensor  # fp32 [H]
    wb_colbias: torch.Tensor
    wo: torch.Tensor         # bf16 [128, 128]
    bo: Optional[torch.Tensor]
    heads: int
    raw_bias: tuple = ()     # (ln_w, ln_b, w_bias) as given: the row-blocked form computes the bias planes first

    @classmethod
    def pack(cls, ln_w, ln_b, w_bias, w_q, w_k, w_v, w_g, b_g, w_o, b_o, heads: int) -> "TriattPacked":
        c = w_q.shape[1]
        if c != 128 or w_q.shape[0] != 128 or heads * 32 != 128:
            raise ValueError("fused triangle attention supports c_z = 128 and 4 heads of 32")
        qs = LOG2E / (32 ** 0.5)
        wq, sq, bq = fold_ln_linear(w_q, ln_w, ln_b, scale=qs)
        wk, sk, bk = fold_ln_linear(w_k, ln_w, ln_b)
        wv, sv, bv = fold_ln_linear(w_v, ln_w, ln_b)
        wg, sg, bg = fold_ln_linear(w_g, ln_w, ln_b, bias=b_g)
        w = torch.cat([wq, wk, wv, wg], 0).contiguous()
        colsum = torch.cat([sq, sk, sv, sg]).contiguous()
        colbias = torch.cat([bq, bk, bv, bg]).contiguous()
        gam = torch.ones(c, device=w_q.device) if ln_w is None else ln_w.detach().float()
        wb = (w_bias.detach().float() * gam[None, :] * LOG2E).contiguous()
        wb_colsum = wb.sum(1).contiguous()
        wb_colbias = torch.zeros(heads, device=w_q.device)
        if ln_b is not None:
            wb_colbias = (w_bias.detach().float() @ ln_b.detach().float()) * LOG2E
        return cls(w, colsum, colbias, wb, wb_colsum, wb_colbias.contiguous(),
                   w_o.detach().to(torch.bfloat16).contiguous(),
                   None if b_o is None else b_o.detach().float().contiguous(), heads, (ln_w, ln_b, w_bias))

    def pointers(self) -> tuple:
        return (self.w.data_ptr(), self.colsum.data_ptr(), self.colbias.data_ptr(), self.wb.data_ptr(), self.wb_colsum.data_ptr(),
                self.wb_colbias.data_ptr(), self.wo.data_ptr(), 0 if self.bo is None else self.bo.data_ptr())


def attention(q, k, v, bias, gate, out, rows: int, Nq: int, Nk: int, H: int, D: int = 32, ldb: int = 0,
              ld_in: int = 0, transpose_out: bool = False, ld_gate: int = 0, mask: Optional[KeyMask] = None):
    """Raw launch of the tcgen05 attention kernel (see csrc/attention_sm100.cu for the layout).
    D is the (padded) head dimension, 32 or 64; ld_in the row stride of q / k / v in elements, ld_gate that of
    the gate (0 = H * D); mask a :class:`KeyMask` over [rows, Nk] or None."""
    st = native.status_tensor(q.device)
    fn = native.lib().ubm_attention_d32 if D == 32 else native.lib().ubm_attention_d64
    if D not in (32, 64):
        raise ValueError("attention kernel supports head dimensions 32 and 64 (pad smaller heads)")
    if mask is not None and (mask.add.shape[0] != rows or mask.add.shape[1] < Nk):
        raise ValueError(f"key mask of shape {tuple(mask.add.shape)} does not cover [{rows}, {Nk}]")
    rc = fn(native.ptr(q), native.ptr(k), native.ptr(v), native.ptr(bias), native.ptr(gate), native.ptr(out),
            native.ptr(None if mask is None else mask.add), native.ptr(None if mask is None else mask.flags), rows,
            Nq, Nk, H, ldb, ld_in, ld_gate, 0 if mask is None else mask.add.stride(0), 1 if transpose_out else 0,
            native.ptr(st), native.current_stream(q.device))
    native.check(rc, f"ubm_attention_d{D}")
    return out


def attention_d32(q, k, v, bias, gate, out, rows, Nq, Nk, H, ldb: int = 0, transpose_out: bool = False,
                  mask: Optional[KeyMask] = None):
    return attention(q, k, v, bias, gate, out, rows, Nq, Nk, H, 32, ldb, 0, transpose_out, mask=mask)


@dataclass
class ApbPacked:
    """Weights of attention-with-pair-bias for the fused path: heads padded to the kernel's head
    dimension (zero rows / columns), q scaled by log2(e)/sqrt(d), q|k|v stacked into one projection."""
    wqkv: torch.Tensor      # bf16 [3*H*Dp, c]
    bqkv: torch.Tensor      # fp32 [3*H*Dp]
    wg: torch.Tensor        # bf16 [H*Dp, c]
    wqkvg: torch.Tensor     # bf16 [4*H*Dp, c]: q|k|v|gate in one projection (sigmoid on the last quarter)
    bqkvg: torch.Tensor     # fp32 [4*H*Dp]
    wo: torch.Tensor        # bf16 [c, H*Dp]
    H: int
    Dp: int

    @classmethod
    def pack(cls, w_q, b_q, w_k, w_v, w_g, w_o, heads: int) -> "ApbPacked":
        c_out, c = w_q.shape
        D = c_out // heads
        Dp = 32 if D <= 32 else 64
        if D > 64:
            raise ValueError("head dimension above 64 is not supported by the attention kernel")

        def pad_rows(W, scale=1.0):
            Wp = torch.zeros((heads, Dp, W.shape[1]), dtype=torch.float32, device=W.device)
            Wp[:, :D] = W.detach().float().view(heads, D, -1) * scale
            return Wp.view(heads * Dp, -1)

        qs = LOG2E / (D ** 0.5)
        wqkv = torch.cat([pad_rows(w_q, qs), pad_rows(w_k), pad_rows(w_v)], 0).to(torch.bfloat16).contiguous()
        bq = torch.zeros((heads, Dp), device=w_q.device)
        if b_q is not None:
            bq[:, :D] = b_q.detach().float().view(heads, D) * qs
        bqkv = torch.cat([bq.view(-1), torch.zeros(2 * heads * Dp, device=w_q.device)]).contiguous()
        wg = pad_rows(w_g).to(torch.bfloat16).contiguous()
        wo = torch.zeros((w_o.shape[0], heads, Dp), dtype=torch.float32, device=w_o.device)
        wo[:, :, :D] = w_o.detach().float().view(w_o.shape[0], heads, D)
        wqkvg = torch.cat([wqkv, wg], 0).contiguous()
        bqkvg = torch.cat([bqkv, torch.zeros(heads * Dp, device=w_q.device)]).contiguous()
        return cls(wqkv, bqkv, wg, wqkvg, bqkvg,
                   wo.view(w_o.shape[0], heads * Dp).to(torch.bfloat16).contiguous(), heads, Dp)


def _one_call(gate: Optional[torch.Tensor], residual: Optional[torch.Tensor], rows: int, cols: int) -> bool:
    """Gate and residual of an output product as the operators that run in one call take them; others go product by product."""
    return (gate is None or (gate.dtype == torch.bfloat16 and gate.dim() == 2 and gate.shape[1] == cols and gate.stride(1) == 1)) \
        and (residual is None or (residual.dtype == torch.bfloat16 and residual.shape == (rows, cols) and residual.is_contiguous()))


def apb_fused(x: torch.Tensor, w: ApbPacked, bias_planes: torch.Tensor, ldb: int,
              out_gate: Optional[torch.Tensor] = None, out_residual: Optional[torch.Tensor] = None,
              mask: Optional[KeyMask] = None, keep: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Gated attention with pair bias on rows x: bf16 [B, N, c]; bias_planes: bf16 [H, N, ldb] holding
    log2(e) * bias (shared by the B rows); mask: key mask over [B, N] or None, or ``keep`` in its place: the mask as the model
    holds it, laid out on the way.
    Returns proj_o(sigmoid(proj_g x) * attention) as [B, N, c];
    with ``out_gate`` ([N, c], shared by the B rows) and ``out_residual`` ([B*N, c]) the output projection's
    epilogue returns residual + gate * projection."""
    B, N, c = x.shape
    HD = w.H * w.Dp
    c_out = w.wo.shape[0]
    if keep is not None:
        keep = KeyMask.readable(keep, (B, N), x.device)
        if keep.shape != (B, N):
            keep, mask = None, KeyMask.lay_out(keep, None, x.device)
    # (the weights' sizes too: the library has only their addresses, one by one the products refuse what does not fit)
    if x.is_cuda and x.dtype == torch.bfloat16 and x.is_contiguous() and w.wqkvg.shape == (4 * HD, c) and w.wo.shape[1] == HD and \
            _one_call(out_gate, out_residual, B * N, c_out):
        dev = x.device
        rows_bytes = 2 * B * N * HD                     # scratch: q | k | v | gate rows, o, additive mask rows and their flags
        ld_mask = add = flags = mask_bytes = keep_ptr = keep_bytes = keep_row = keep_key = 0
        if keep is not None:
            ld_mask = ceil_to(N, MASK_STEP)
            mask_bytes = B * (2 * ld_mask + ld_mask // MASK_STEP)
        scratch = torch.empty(5 * rows_bytes + mask_bytes, dtype=torch.uint8, device=dev)
        qkvg = scratch.data_ptr()
        if keep is not None:
            add = qkvg + 5 * rows_bytes
            flags = add + 2 * B * ld_mask
            keep_ptr, keep_bytes = keep.data_ptr(), keep.element_size()
            keep_row, keep_key = keep.stride()
            native.add_launches(1, "ubm_key_mask")
        elif mask is not None:
            if mask.add.shape[0] != B or mask.add.shape[1] < N:
                raise ValueError(f"key mask of shape {tuple(mask.add.shape)} does not cover [{B}, {N}]")
            add, flags, ld_mask = mask.add.data_ptr(), mask.flags.data_ptr(), mask.add.stride(0)
        out = torch.empty((B, N, c_out), dtype=torch.bfloat16, device=dev)
        rc = native.lib().ubm_apb(_APB_ARGS.pack(
            x.data_ptr(), w.wqkvg.data_ptr(), w.bqkvg.data_ptr(), w.wo.data_ptr(), native.ptr(bias_planes), ldb, keep_ptr, keep_bytes,
            keep_row, keep_key, add, flags, ld_mask, native.ptr(out_gate), 0 if out_gate is None else out_gate.stride(0),
            0 if out_gate is None else out_gate.shape[0], native.ptr(out_residual), qkvg, qkvg + 4 * rows_bytes, out.data_ptr(),
            B, N, c, c_out, w.H, w.Dp, native.status_tensor(dev).data_ptr(), native.current_stream(dev)))
        native.check(rc, "ubm_apb")
        return out
    if keep is not None:
        mask = KeyMask.lay_out(keep, None, x.device)
    x2 = x.reshape(B * N, c)
    # q | k | v | gate from one GEMM (sigmoid on the gate columns); the attention kernel reads all four as column
    # slices of its output
    qkvg = _gemm.gemm(x2, w.wqkvg, bias=w.bqkvg, act="sigmoid", act_from=3 * HD)
    o = torch.empty((B * N, HD), dtype=torch.bfloat16, device=x.device)
    attention(qkvg[:, :HD], qkvg[:, HD:2 * HD], qkvg[:, 2 * HD:3 * HD], bias_planes, qkvg[:, 3 * HD:], o, rows=B,
              Nq=N, Nk=N, H=w.H, D=w.Dp, ldb=ldb, ld_in=4 * HD, ld_gate=4 * HD, mask=mask)
    return _gemm.gemm(o, w.wo, gate=out_gate, residual=out_residual).view(B, N, -1)


def single_track(s: torch.Tensor, z: torch.Tensor, keep: Optional[torch.Tensor], norm: tuple, bias: tuple, w: ApbPacked,
                 norm2: tuple, w12: torch.Tensor, w3: torch.Tensor) -> torch.Tensor:
    """The single track of a Pairformer layer from one call: s + attention of its norm with the bias from z, then + transition, sums in
    fp32.  s: bf16 [1, N, c], z: bf16 [1, N, N, 128], contiguous; keep: [1, N] of a type :meth:`KeyMask.readable` leaves alone, or None;
    norms as (fp32 gamma, beta or None, eps); bias: :func:`ops.rows._head_bias_weights`; w12, w3 as :func:`transition_rows` takes them."""
    N, c = s.shape[1:]
    dev = s.device
    hidden = w3.shape[1]
    if w.wqkvg.shape != (4 * w.H * w.Dp, c) or w.wo.shape != (c, w.H * w.Dp) or w12.shape != (2 * hidden, c) or w3.shape[0] != c or \
            bias[0].shape != (w.H, 128) or z.shape != (1, N, N, 128):
        raise ValueError(f"single_track: weights of other sizes than {tuple(s.shape)} and {tuple(z.shape)} take")
    ldb, ld_mask, HD = ceil_to(N, 8), ceil_to(N, MASK_STEP), w.H * w.Dp
    row = 2 * N * c                                         # one [N, c] in bf16
    sizes = (2 * w.H * N * ldb, row, 8 * N * HD, 2 * N * HD, row, 2 * row, row, 2 * N * hidden, 2 * ld_mask, ld_mask // MASK_STEP)
    at = [0]
    for n in sizes:
        at.append(at[-1] + ceil_to(n, 256))
    scratch = torch.empty(at[-1], dtype=torch.uint8, device=dev)
    p = scratch.data_ptr()
    planes, n, qkvg, o, upd, s32, x, h, add, flags = (p + a for a in at[:-1])
    keep_ptr = keep_bytes = keep_key = 0
    if keep is None:
        add = flags = ld_mask = 0
    else:
        keep_ptr, keep_bytes, keep_key = keep.data_ptr(), keep.element_size(), keep.stride(1)
        native.add_launches(1, "ubm_key_mask")
    out = torch.empty_like(s)
    ptr = native.ptr
    rc = native.lib().ubm_single_track(_SINGLE_TRACK_ARGS.pack(
        s.data_ptr(), z.data_ptr(), ptr(norm[0]), ptr(norm[1]), *(t.data_ptr() for t in bias), w.wqkvg.data_ptr(), w.bqkvg.data_ptr(),
        w.wo.data_ptr(), ptr(norm2[0]), ptr(norm2[1]), w12.data_ptr(), w3.data_ptr(), norm[2], norm2[2], keep_ptr, keep_bytes, keep_key,
        add, flags, ld_mask, planes, n, qkvg, o, upd, s32, x, h, out.data_ptr(), N, ldb, c, w.H, w.Dp, hidden,
        native.status_tensor(dev).data_ptr(), native.current_stream(dev)))
    native.check(rc, "ubm_single_track")
    return out


def _triatt_blocked(z, w: TriattPacked, starting: bool, residual: bool, out, ws: dict, mask, rb: int):
    """Row-blocked triangle attention: the per-head bias planes of the whole pair tensor first (one pass of a row
    kernel; transposed for the ending node), then projection -> attention -> output projection for ``rb``
    attention rows at a time, so q | k | v | gate | o exist for one block only.  For the ending node an attention
    row is a column of z: the block's columns are gathered to rows before the projection and the update is
    added back to those columns."""
    from . import rows as _rows
    N = z.shape[0]
    Np = ceil_to(N, 8)
    dev = z.device
    key = ("triatt_blocked", N, rb, dev)
    if key not in ws:
        ws[key] = (torch.empty((5, rb * N, 128), dtype=torch.bfloat16, device=dev),
                   torch.zeros((w.heads, N, Np), dtype=torch.bfloat16, device=dev),
                   torch.zeros((w.heads, rb, Np), dtype=torch.bfloat16, device=dev))
    qkvgo, hb, hb_scratch = ws[key]
    ln_w, ln_b, w_bias = w.raw_bias
    _rows.pair_head_bias(z, ln_w, ln_b, w_bias, scale=LOG2E, transpose=not starting, out=hb)
    st = native.status_tensor(dev)
    stream = native.current_stream(dev)
    lib = native.lib()
    out = torch.empty_like(z) if out is None else out
    for r0 in range(0, N, rb):
        r1 = min(N, r0 + rb)
        R = r1 - r0
        src = z[r0:r1] if starting else z[:, r0:r1].transpose(0, 1).contiguous()
        q, k, v, g, og = (qkvgo[i][: R * N] for i in range(5))
        rc = lib.ubm_triatt_proj_rows(native.ptr(src), native.ptr(w.w), native.ptr(w.colsum), native.ptr(w.colbias),
                                      native.ptr(w.wb), native.ptr(w.wb_colsum), native.ptr(w.wb_colbias),
                                      native.ptr(q), native.ptr(k), native.ptr(v), native.ptr(g),
                                      native.ptr(hb_scratch), 0, R, rb, N, Np, w.heads, 0, native.ptr(st), stream)
        native.check(rc, "ubm_triatt_proj_rows")
        km = None if mask is None else KeyMask(mask.add[r0:r1], mask.flags[r0:r1])
        attention_d32(q, k, v, hb, g, og, rows=R, Nq=N, Nk=N, H=w.heads, ldb=Np, mask=km)
        if starting:
            _gemm.gemm(og, w.wo, bias=w.bo, residual=z[r0:r1].view(R * N, 128) if residual else None,
                       out=out[r0:r1].view(R * N, 128))
        else:
            upd = _gemm.gemm(og, w.wo, bias=w.bo).view(R, N, 128).transpose(0, 1)
            out[:, r0:r1] = (z[:, r0:r1] + upd) if residual else upd
    return out


def _triatt_scratch(ws: dict, N: int, Np: int, heads: int, dev) -> tuple:
    key = ("triatt", N, dev)
    if key not in ws:
        ws[key] = (torch.empty((5, N * N, 128), dtype=torch.bfloat16, device=dev),
                   torch.zeros((heads, N, Np), dtype=torch.bfloat16, device=dev))
    return ws[key]


def _triatt_into(z, w: TriattPacked, starting: bool, residual: bool, out, ws: dict, mask):
    """The launches of :func:`triangle_attention_fused` one by one, for an ``out`` that only the output product can write: fp32, or
    rows of [N * N, 128] in a wider buffer."""
    N, dev = z.shape[0], z.device
    Np = ceil_to(N, 8)
    to = out.view(N * N, 128)
    if out.dtype not in (torch.bfloat16, torch.float32) or out.device != dev:
        raise ValueError(f"triangle attention writes bf16 or fp32 on {dev}, not {out.dtype} on {out.device}")
    qkvgo, hb = _triatt_scratch(ws, N, Np, w.heads, dev)
    q, k, v, g, og = qkvgo
    rc = native.lib().ubm_triatt_proj(native.ptr(z), native.ptr(w.w), native.ptr(w.colsum), native.ptr(w.colbias), native.ptr(w.wb),
                                      native.ptr(w.wb_colsum), native.ptr(w.wb_colbias), native.ptr(q), native.ptr(k), native.ptr(v),
                                      native.ptr(g), native.ptr(hb), 0, N, Np, w.heads, 0 if starting else 1,
                                      native.ptr(native.status_tensor(dev)), native.current_stream(dev))
    native.check(rc, "ubm_triatt_proj")
    attention_d32(q, k, v, hb, g, og, rows=N, Nq=N, Nk=N, H=w.heads, ldb=Np, transpose_out=not starting, mask=mask)
    _gemm.gemm(og, w.wo, bias=w.bo, residual=z.view(N * N, 128) if residual else None, out=to)
    return out


def triangle_attention_fused(z: torch.Tensor, w: TriattPacked, starting: bool, residual: bool = True,
                             out: Optional[torch.Tensor] = None, workspace: Optional[dict] = None,
                             mask: Optional[KeyMask] = None, keep: Optional[torch.Tensor] = None) -> torch.Tensor:
    """z: bf16 [N, N, 128] contiguous; mask: key mask over [attention row, key] (for the ending node the
    attention rows are the columns of z, so the caller packs the transposed pair mask), or ``keep`` in its place: the mask as
    the model holds it, laid out on the way.  Three launches:
    projection (LN folded, q|k|v|gate rows + head bias planes, written at the transposed pair index for the
    ending node) -> attention -> output projection with residual."""
    if z.dtype != torch.bfloat16 or z.dim() != 3 or z.shape[-1] != 128 or not z.is_contiguous():
        raise ValueError("triangle_attention_fused expects a contiguous bf16 [N, N, 128] tensor")
    N = z.shape[0]
    Np = ceil_to(N, 8)
    dev = z.device
    ws = workspace if workspace is not None else {}
    rb = int(ws.get("row_block", 0) or 0)
    if 0 < rb < N:
        if keep is not None:
            mask = KeyMask.lay_out(keep, (N, N), dev)
        return _triatt_blocked(z, w, starting, residual, out, ws, mask, rb)
    if out is not None and (out.dtype != torch.bfloat16 or not out.is_contiguous()):
        if keep is not None:
            mask = KeyMask.lay_out(keep, (N, N), dev)
        return _triatt_into(z, w, starting, residual, out, ws, mask)
    out = _result(out, z)
    add = flags = keep_ptr = keep_bytes = keep_row = keep_key = ld_mask = 0
    if keep is not None:
        keep = KeyMask.readable(keep, (N, N), dev)
        if keep.shape != (N, N):
            keep, mask = None, KeyMask.lay_out(keep, None, dev)
    if keep is not None:
        ld_mask = ceil_to(N, MASK_STEP)
        laid = torch.empty(N * (2 * ld_mask + ld_mask // MASK_STEP), dtype=torch.uint8, device=dev)     # additive rows, then flags
        add, keep_ptr, keep_bytes = laid.data_ptr(), keep.data_ptr(), keep.element_size()
        flags = add + 2 * N * ld_mask
        keep_row, keep_key = keep.stride()
        native.add_launches(1, "ubm_key_mask")
    elif mask is not None:
        if mask.add.shape[0] != N or mask.add.shape[1] < N:
            raise ValueError(f"key mask of shape {tuple(mask.add.shape)} does not cover [{N}, {N}]")
        add, flags, ld_mask = mask.add.data_ptr(), mask.flags.data_ptr(), mask.add.stride(0)
    qkvgo, hb = _triatt_scratch(ws, N, Np, w.heads, dev)
    rc = native.lib().ubm_triatt(_TRIATT_ARGS.pack(
        z.data_ptr(), keep_ptr, keep_bytes, keep_row, keep_key, add, flags, ld_mask, *w.pointers(), qkvgo.data_ptr(), hb.data_ptr(), out.data_ptr(), N, Np, w.heads,
        1 if starting else 0, 1 if residual else 0, native.status_tensor(dev).data_ptr(), native.current_stream(dev)))
    native.check(rc, "ubm_triatt")
    return out


def pair_track(z: torch.Tensor, mask: Optional[torch.Tensor], tm_out: TrimulPacked, tm_in: TrimulPacked, ta_start: TriattPacked,
               ta_end: TriattPacked, tr: TransitionPacked, workspace: dict) -> torch.Tensor:
    """The five pair operators of a Pairformer layer, each with its residual, from one call.  z: bf16 [1, N, N, 128] contiguous; mask:
    bf16 [1, N, N] contiguous or None."""
    N, dev = z.shape[1], z.device
    Np, bias_row = ceil_to(N, PLANE_ROW), ceil_to(N, 8)
    planes, x = _trimul_scratch(workspace, N, Np, dev)
    qkvgo, hb = _triatt_scratch(workspace, N, bias_row, ta_start.heads, dev)
    out, other = torch.empty_like(z), torch.empty_like(z)
    add = flags = ld_mask = mask_ptr = 0
    if mask is not None:
        ld_mask, mask_ptr = ceil_to(N, MASK_STEP), mask.data_ptr()
        laid = torch.empty(N * (2 * ld_mask + ld_mask // MASK_STEP), dtype=torch.uint8, device=dev)     # additive rows, then flags
        add = laid.data_ptr()
        flags = add + 2 * N * ld_mask
        native.add_launches(2, "ubm_key_mask")
    rc = native.lib().ubm_pair_track(_PAIR_TRACK_ARGS.pack(
        z.data_ptr(), out.data_ptr(), other.data_ptr(), mask_ptr, add, flags, ld_mask, *tm_out.pointers(), *tm_in.pointers(),
        *ta_start.pointers(), *ta_end.pointers(), tr.wab.data_ptr(), tr.wo.data_ptr(), tr.colsum.data_ptr(), tr.colbias.data_ptr(),
        tr.hidden, planes.data_ptr(), x.data_ptr(), qkvgo.data_ptr(), hb.data_ptr(), N, Np, bias_row, ta_start.heads,
        native.status_tensor(dev).data_ptr(), native.current_stream(dev)))
    native.check(rc, "ubm_pair_track")
    return out


# ------------------------------------------------------------------------------------------
native.declare("ubm_pair_weighted_averaging", [c_void_p] * 3 + [c_int] + [c_void_p, c_int] * 4 + [c_void_p] * 5 +
               [c_int] * 3 + [c_float] + [c_void_p] * 2)


@dataclass
class PwaPacked:
    """Parameters of a pair-weighted averaging as the kernels take them.  Nothing is folded ahead: each call folds the
    LayerNorm into the two projections (one launch over 64 KB), so a weight written by any route counts."""
    args: tuple              # address and fp32 flag of the value and gate projections and the LayerNorm's weight and bias
    held: tuple              # the tensors behind the addresses
    wo: torch.Tensor         # bf16 [64, 256]
    eps: float

    @classmethod
    def pack(cls, norm_w, norm_b, w_m, w_g, w_o, eps: float) -> "PwaPacked":
        """Parameters bf16 or fp32 (others are converted); norm_w / norm_b may be None."""
        if w_m.shape != (256, 64) or w_g.shape != (256, 64) or w_o.shape != (64, 256):
            raise ValueError("fused pair-weighted averaging supports c_m = 64 and 8 heads of 32")
        dev, args, held = w_m.device, [], []
        for t in (w_m, w_g, norm_w, norm_b):
            if t is None:
                args += (0, 0)
                continue
            if t.device != dev or t.shape[-1] != 64:
                raise ValueError("fused pair-weighted averaging: parameters of one device and 64 channels")
            fp32 = t.dtype != torch.bfloat16
            if fp32 or not t.is_contiguous():
                t = t.detach().to(torch.float32 if fp32 else t.dtype).contiguous()
            held.append(t)
            args += (t.data_ptr(), 1 if fp32 else 0)
        if w_o.dtype != torch.bfloat16 or not w_o.is_contiguous():
            w_o = w_o.detach().to(torch.bfloat16).contiguous()
        return cls(tuple(args), tuple(held), w_o, float(eps))


def pair_weighted_averaging_fused(m: torch.Tensor, b: torch.Tensor, mask: Optional[torch.Tensor],
                                  w: PwaPacked) -> torch.Tensor:
    """m: bf16 [S, N, 64] contiguous; b: bf16 [8, N, N], a view of planes with row stride Np (from ``pair_head_bias``),
    overwritten; mask: [N, N] (1 = keep) or None.  Returns proj_o(sigmoid(proj_g n) * softmax(b + mask) v), n = LN(m)."""
    S, N, c = m.shape
    Np = b.stride(1)
    if m.dtype != torch.bfloat16 or c != 64 or not m.is_contiguous() or b.shape != (8, N, N) or b.stride(0) != N * Np:
        raise ValueError("pair_weighted_averaging_fused expects contiguous bf16 [S, N, 64] and planes of 8 heads")
    dev = m.device
    if b.device != dev or w.wo.device != dev or (mask is not None and mask.device != dev):
        raise ValueError("pair_weighted_averaging_fused: rows, bias planes, weights and mask live on one GPU")
    if mask is not None and mask.dtype != torch.bfloat16:
        mask = mask.float()
    mk = None if mask is None else mask.expand(N, N).contiguous()
    fold = torch.empty(2 * 256 * 64 * 2 + 4 * 256 * 4, dtype=torch.uint8, device=dev)
    v = torch.empty((8, S * 32, Np), dtype=torch.bfloat16, device=dev)
    o = torch.empty((N, S, 256), dtype=torch.bfloat16, device=dev)
    out = torch.empty_like(m)
    rc = native.lib().ubm_pair_weighted_averaging(
        m.data_ptr(), b.data_ptr(), 0 if mk is None else mk.data_ptr(), 1 if mk is not None and mk.dtype == torch.bfloat16
        else 0, *w.args, w.wo.data_ptr(), fold.data_ptr(), v.data_ptr(), o.data_ptr(), out.data_ptr(), S, N, Np, w.eps,
        native.status_tensor(dev).data_ptr(), native.current_stream(dev))
    native.check(rc, "ubm_pair_weighted_averaging")
    return out


# ------------------------------------------------------------------------------------------
native.declare("ubm_window_attention", [c_void_p] * 6 + [c_int, c_int, c_int, c_ll, c_int, c_void_p])
native.declare("ubm_window_attention_tc", [c_void_p] * 6 + [c_int, c_int, c_int, c_ll, c_int, c_void_p, c_void_p])

WINDOW_KERNEL = "tc"     # "tc": matrix instructions (4 heads at 128 channels: ops.atom; else the tcgen05 kernel); "simt": CUDA cores


def window_attention_fused(x: torch.Tensor, w: ApbPacked, bias: Optional[torch.Tensor],
                           out_gate: Optional[torch.Tensor] = None,
                           out_residual: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Gated atom attention in 32 x 128 windows.  x: bf16 [B, A, c] (A a multiple of 32); w: packed projections with
    4 x 32 heads; bias: bf16 [1 or B, H, A/32, 32, 128] already multiplied by log2(e).  Returns [B, A, c]."""
    B, A, c = x.shape
    if w.Dp != 32:
        raise ValueError("window attention supports head dimension 32")
    HD = w.H * 32
    x2 = x.reshape(B * A, c)
    from . import atom
    if atom._window_serves(w, bias, B, A, c) and (out_gate is None or atom._gate_of(out_gate, B * A) is not None) and \
            (out_residual is None or (atom._plain(out_residual) and out_residual.numel() == B * A * c)):
        qkvg = _gemm.gemm(x2, w.wqkvg, bias=w.bqkvg, act="sigmoid", act_from=3 * HD)
        return atom.window_layer(qkvg, w, bias, out_gate, out_residual, B, A)
    qkv = _gemm.gemm(x2, w.wqkv, bias=w.bqkv)
    g = _gemm.gemm(x2, w.wg, act="sigmoid")
    o = torch.empty((B * A, HD), dtype=torch.bfloat16, device=x.device)
    if WINDOW_KERNEL == "tc":
        rc = native.lib().ubm_window_attention_tc(native.ptr(qkv), native.ptr(qkv) + HD * 2,
                                                  native.ptr(qkv) + 2 * HD * 2, native.ptr(bias), native.ptr(g),
                                                  native.ptr(o), B, A, w.H, 3 * HD,
                                                  1 if bias is None else bias.shape[0],
                                                  native.ptr(native.status_tensor(x.device)),
                                                  native.current_stream(x.device))
        native.check(rc, "ubm_window_attention_tc")
    else:
        rc = native.lib().ubm_window_attention(native.ptr(qkv), native.ptr(qkv) + HD * 2,
                                               native.ptr(qkv) + 2 * HD * 2, native.ptr(bias), native.ptr(g),
                                               native.ptr(o), B, A, w.H, 3 * HD,
                                               1 if bias is None else bias.shape[0], native.current_stream(x.device))
        native.check(rc, "ubm_window_attention")
    return _gemm.gemm(o, w.wo, gate=out_gate, residual=out_residual).view(B, A, -1)
