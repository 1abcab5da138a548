"""Kernels of the atom-transformer layer against float64, at the edges of their tiles: windows that reach past either end, an odd
last window, row tiles that end inside a sample, conditioning shared by the samples or their own, gates that are column slices."""
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _rand(g, *shape, scale=1.0):
    return (torch.randn(shape, device="cuda", generator=g) * scale).to(BF)


def _conditions(g, rows, wide):
    """scale, shift, gate (a sigmoid already); ``wide``: column slices of one buffer."""
    if wide:
        buf = _rand(g, rows, 5 * 128)
        gates = torch.sigmoid(buf.float()).to(BF)
        return buf[:, 128:256], buf[:, 256:384], gates[:, 384:512]
    return _rand(g, rows, 128), _rand(g, rows, 128), torch.sigmoid(_rand(g, rows, 128).float()).to(BF)


def _norm(a, sc, sh):
    n = F.layer_norm(a.double(), (128,), eps=1e-5).view(-1, sc.shape[0], 128)
    return (torch.sigmoid(sc.double()) * n + sh.double()).view(a.shape)


def _err(x, ref):
    return ((x.double() - ref).norm() / ref.norm()).item()


def _check(out, general, ref, what):
    """No further from float64 than one product at a time: both round the same intermediates to bf16, in the same places; the rest
    (order of fp32 sums, 2^-24 each) is far below a twentieth of that."""
    from uplifting_biomolecular_modeling_b200.ops import native
    torch.cuda.synchronize()
    native.raise_on_status("cuda", what)
    assert torch.isfinite(out).all()
    e, e0 = _err(out, ref), _err(general, ref)
    assert e <= 1.05 * e0 + 1e-5, (what, e, e0)


@pytest.mark.parametrize("B,A", [(1, 32), (2, 64), (3, 96), (1, 160), (5, 352), (2, 4064)])
@pytest.mark.parametrize("own,wide", [(False, False), (False, True), (True, False)])
def test_attention_half(B, A, own, wide, monkeypatch):
    from uplifting_biomolecular_modeling_b200.models import diffusion
    from uplifting_biomolecular_modeling_b200.ops import atom, native, pair, rows
    g = torch.Generator(device="cuda").manual_seed(A + B)
    a = _rand(g, B, A, 128, scale=1.5)
    sc, sh, gate = _conditions(g, B * A if own else A, wide)
    ws = [_rand(g, 128, 128, scale=128 ** -0.5) for _ in range(5)]
    bq = _rand(g, 128, scale=0.3)
    w = pair.ApbPacked.pack(ws[0], bq, ws[1], ws[2], ws[3], ws[4], 4)
    bias = _rand(g, B if own else 1, 4, A // 32, 32, 128)
    data = diffusion.WindowBias(bias).data
    n = _norm(a, sc, sh)
    q, k, v, gt = ((n @ m.double().T) for m in ws[:4])
    q = q + bq.double()
    idx = torch.arange(A // 32, device="cuda")[:, None] * 32 - 48 + torch.arange(128, device="cuda")
    ok = (idx >= 0) & (idx < A)
    at = idx.clamp(0, A - 1)
    heads = lambda x: x.view(B, A, 4, 32)  # noqa: E731
    s = torch.einsum("bwqhd,bwkhd->bhwqk", heads(q).view(B, -1, 32, 4, 32), heads(k)[:, at]) / math.sqrt(32) + data.double() / 1.4426950408889634
    p = torch.softmax(s.masked_fill(~ok[None, None, :, None, :], float("-inf")), -1)
    o = torch.einsum("bhwqk,bwkhd->bwqhd", p, heads(v)[:, at]).reshape(B, A, 128) * torch.sigmoid(gt)
    ref = a.double() + (gate.double() * (o @ ws[4].double().T).view(-1, gate.shape[0], 128)).view(B, A, 128)
    native.reset_launch_count()
    out = atom.attention(a, sc, sh, w, data, gate)
    assert native.launch_counts() == {"ubm_atom_qkvg": 1, "ubm_window_layer": 1}
    x = rows.adaln_rows(a, sc, sh)
    mid = pair.window_attention_fused(x, w, data, out_gate=gate, out_residual=a.view(B * A, 128))
    plain = pair.window_attention_fused(x, w, data)          # neither gate nor residual
    monkeypatch.setattr(atom, "_window_serves", lambda *k: False)
    general = atom.attention(a, sc, sh, w, data, gate)
    _check(out, general, ref, "attention half")
    _check(mid, general, ref, "window layer behind the GEMM")
    _check(plain, pair.window_attention_fused(x, w, data), (o @ ws[4].double().T), "window layer alone")


@pytest.mark.parametrize("runs,rows_", [(1, 128), (3, 129), (5, 333), (1, 1000), (2, 20000)])
@pytest.mark.parametrize("hidden,wide", [(256, False), (256, True), (32, False), (96, True)])
def test_transition_half(runs, rows_, hidden, wide):
    from uplifting_biomolecular_modeling_b200.ops import atom, gemm, native
    g = torch.Generator(device="cuda").manual_seed(rows_ + hidden)
    a = _rand(g, runs, rows_, 128, scale=1.5)
    sc, sh, gate = _conditions(g, rows_, wide)
    wg, wv, wu = (_rand(g, hidden, 128, scale=128 ** -0.5) for _ in range(3))
    wo = _rand(g, 128, hidden, scale=hidden ** -0.5)
    n = _norm(a, sc, sh)
    h = F.silu(n @ wg.double().T) * (n @ wv.double().T) * (n @ wu.double().T)
    ref = a.double() + gate.double() * (h @ wo.double().T)
    native.reset_launch_count()
    out = atom.transition(a, sc, sh, gate, gemm.pack_swiglu3(wg, wv, wu), wo)
    assert native.launch_counts() == {"ubm_cond_transition": 1}
    general = atom.transition(a, sc, sh, gate, torch.cat([wg, wv, wu]).contiguous(), wo, packed=False)
    _check(out, general, ref, "conditioned transition")


def test_forms_the_kernels_do_not_take():
    """Rows off 16 bytes, runs shorter than a tile, other widths: one product at a time, same result."""
    from uplifting_biomolecular_modeling_b200.ops import atom, gemm, native
    g = torch.Generator(device="cuda").manual_seed(3)
    sc, sh, gate = _conditions(g, 64, False)
    a = _rand(g, 4, 64, 128)
    wg, wv, wu = (_rand(g, 64, 128, scale=128 ** -0.5) for _ in range(3))
    wo, w_in = _rand(g, 128, 64, scale=0.125), None
    w_in = gemm.pack_swiglu3(wg, wv, wu)
    n = _norm(a, sc, sh)
    h = F.silu(n @ wg.double().T) * (n @ wv.double().T) * (n @ wu.double().T)
    ref = a.double() + gate.double() * (h @ wo.double().T)
    native.reset_launch_count()
    out = atom.transition(a, sc, sh, gate, w_in, wo)
    assert "ubm_cond_transition" not in native.launch_counts()
    assert _err(out, ref) < 6e-3          # four bf16 roundings of 2^-9 at most, one behind the other
