"""Operators that run from one call of the library: the same results, bit for bit, as launch by launch, over the masks, strides and
epilogue operands that either form takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _rand(g, *shape):
    return torch.randn(shape, device="cuda", generator=g).to(BF)


def _module(build, seed=0):
    from uplifting_biomolecular_modeling_b200.models import pairformer
    torch.manual_seed(seed)
    m = build(pairformer).cuda().to(BF).eval().requires_grad_(False)
    pairformer.set_impl(m, "fused")
    return m


@pytest.mark.parametrize("N", [16, 77, 128, 201])
@pytest.mark.parametrize("outgoing", [True, False])
def test_triangle_multiplication_masks(N, outgoing):
    """bf16 masks are read in place, others converted; a strided one is copied first."""
    m = _module(lambda p: p.TriangleMultiplication(128, outgoing))
    g = torch.Generator(device="cuda").manual_seed(N)
    z = _rand(g, 1, N, N, 128)
    mask = (torch.rand((1, N, N), device="cuda", generator=g) < 0.8).to(BF) * 0.75
    wide = torch.zeros((1, N, N + 3), device="cuda", dtype=BF)
    wide[:, :, :N] = mask
    ref = m(z, mask.float(), residual=True)
    for other in (mask, wide[:, :, :N], mask.double()):
        assert torch.equal(m(z, other, residual=True), ref)
    assert not torch.equal(m(z, None, residual=True), ref)


@pytest.mark.parametrize("N", [16, 77, 130])
@pytest.mark.parametrize("starting", [True, False])
def test_triangle_attention_masks(N, starting):
    from uplifting_biomolecular_modeling_b200.ops import pair
    m = _module(lambda p: p.TriangleAttention(starting=starting))
    g = torch.Generator(device="cuda").manual_seed(N)
    z = _rand(g, 1, N, N, 128)
    keep = torch.rand((1, N, N), device="cuda", generator=g) < 0.7
    keep[:, :, 0] = keep[:, 0, :] = True
    first = m(z, keep.to(BF), residual=True)
    laid = pair.KeyMask.lay_out(keep[0] if starting else keep[0].t(), (N, N), z.device)
    ref = pair.triangle_attention_fused(z[0], m._packed, starting, residual=True, mask=laid)[None]
    assert torch.equal(first, ref)
    for other in (keep, keep.float(), keep.double(), keep.to(BF).transpose(1, 2).contiguous().transpose(1, 2)):
        assert torch.equal(m(z, other, residual=True), ref)
    one = torch.ones((1, 1, N), device="cuda", dtype=BF)                    # broadcast over the rows
    assert torch.equal(m(z, one, residual=False), m(z, torch.ones_like(keep), residual=False))
    with pytest.raises(ValueError):
        pair.triangle_attention_fused(z[0], m._packed, starting, keep=torch.ones((N - 1, N), device="cuda"))


@pytest.mark.parametrize("starting", [True, False])
@pytest.mark.parametrize("N", [16, 77])
def test_triangle_attention_outputs_of_other_forms(N, starting):
    """An fp32 output holds the sums before their rounding, rows of a wider buffer the result itself; the rest of it is left alone."""
    from uplifting_biomolecular_modeling_b200.ops import pair
    m = _module(lambda p: p.TriangleAttention(starting=starting))
    g = torch.Generator(device="cuda").manual_seed(N)
    z = _rand(g, 1, N, N, 128)
    keep = (torch.rand((N, N), device="cuda", generator=g) < 0.7) | torch.eye(N, device="cuda", dtype=torch.bool)
    m(z)                                                                    # packs the weights
    ref = pair.triangle_attention_fused(z[0], m._packed, starting, keep=keep)
    wide = torch.full((N, N, 192), 7.0, device="cuda", dtype=BF)
    pair.triangle_attention_fused(z[0], m._packed, starting, keep=keep, out=wide[:, :, :128])
    assert torch.equal(wide[:, :, :128], ref) and bool((wide[:, :, 128:] == 7).all())
    full = torch.empty((N, N, 128), device="cuda")
    pair.triangle_attention_fused(z[0], m._packed, starting, keep=keep, out=full)
    assert torch.equal(full.to(BF), ref) and not torch.equal(full, ref.float())


@pytest.mark.parametrize("B,N,c,heads", [(1, 5, 384, 16), (2, 137, 384, 16), (3, 200, 768, 16), (1, 64, 128, 4)])
@pytest.mark.parametrize("epilogue", ["plain", "gate", "slice"])
@pytest.mark.parametrize("masked", [False, True])
def test_pair_bias_attention(B, N, c, heads, epilogue, masked, monkeypatch):
    from uplifting_biomolecular_modeling_b200.ops import pair
    g = torch.Generator(device="cuda").manual_seed(N + c)
    w = pair.ApbPacked.pack(*(_rand(g, c, c) * c ** -0.5 if i != 1 else _rand(g, c) for i in range(6)), heads)
    x = _rand(g, B, N, c)
    ldb = (N + 7) // 8 * 8
    planes = _rand(g, heads, N, ldb)
    keep = (torch.rand((B, N), device="cuda", generator=g) < 0.8).to(BF) if masked else None
    mask = pair.KeyMask.lay_out(keep) if masked else None
    gate = residual = None
    if epilogue != "plain":
        gate = torch.sigmoid(_rand(g, N, c + 64).float()).to(BF)
        gate = gate[:, 64:] if epilogue == "slice" else gate[:, 64:].contiguous()
        residual = _rand(g, B * N, c)
    out = pair.apb_fused(x, w, planes, ldb, gate, residual, mask)
    assert torch.equal(out, pair.apb_fused(x, w, planes, ldb, gate, residual, keep=keep))
    monkeypatch.setattr(pair, "_one_call", lambda *a: False)
    assert torch.equal(out, pair.apb_fused(x, w, planes, ldb, gate, residual, mask))
    assert torch.equal(out, pair.apb_fused(x, w, planes, ldb, gate, residual, keep=keep))


@pytest.mark.parametrize("R,dim,hidden,out_dim", [(1, 384, 1536, 384), (137, 384, 1536, 384), (1000, 64, 256, 64), (130, 256, 96, 128)])
@pytest.mark.parametrize("residual", [False, True])
def test_transition_of_other_widths(R, dim, hidden, out_dim, residual):
    from uplifting_biomolecular_modeling_b200.ops import gemm, pair, rows
    g = torch.Generator(device="cuda").manual_seed(R + dim)
    x, nw, nb = _rand(g, R, dim), _rand(g, dim), _rand(g, dim)
    w12 = gemm.pack_swiglu(_rand(g, hidden, dim) * dim ** -0.5, _rand(g, hidden, dim) * dim ** -0.5)
    w3 = _rand(g, out_dim, hidden) * hidden ** -0.5
    residual = residual and out_dim == dim
    out = pair.transition_rows(x, nw, nb, 1e-5, w12, w3, residual)
    h = gemm.gemm(rows.layernorm_rows(x, nw, nb, 1e-5), w12, act="swiglu")
    assert torch.equal(out, gemm.gemm(h, w3, residual=x if residual else None))


@pytest.mark.parametrize("N", [16, 48, 137, 200])
@pytest.mark.parametrize("masked", [False, True])
def test_pair_track_in_one_call(N, masked, monkeypatch):
    """The same bits, ledger and launch counts as operator by operator."""
    from uplifting_biomolecular_modeling_b200.core import counters
    from uplifting_biomolecular_modeling_b200.models import pairformer
    from uplifting_biomolecular_modeling_b200.ops import native
    m = _module(lambda p: p.PairformerLayer())
    g = torch.Generator(device="cuda").manual_seed(N)
    z = _rand(g, 1, N, N, 128)
    kept = z.clone()
    keep = torch.ones((1, N), device="cuda", dtype=BF)
    keep[:, N - N // 8:] = 0
    mask = keep[:, :, None] * keep[:, None, :] if masked else None
    served = lambda: {k: counters.BOOK.find(k).served for k in ("fused_trimul", "fused_triatt", "fused_transition")}  # noqa: E731
    ref = m.pair_update(z, mask)                       # packs the weights, operator by operator
    calls = []
    for one in (False, True):
        with monkeypatch.context() as mp:
            if not one:
                mp.setattr(pairformer.PairformerLayer, "_pair_track", lambda self, z, mask: None)
            before = served()
            native.reset_launch_count()
            out = m.pair_update(z, mask)
            calls.append((native.launch_counts(), {k: v - before[k] for k, v in served().items()}))
        assert torch.equal(out, ref) and torch.equal(z, kept)
    assert calls[0] == calls[1]
    assert m._pair_track(z, mask) is not None


def test_what_keeps_the_pair_track_apart():
    """A hook, another forward, row blocks, a mask of another type or strides, a batch: operator by operator, same result."""
    from uplifting_biomolecular_modeling_b200.models import pairformer
    N = 32
    m = _module(lambda p: p.PairformerLayer())
    g = torch.Generator(device="cuda").manual_seed(1)
    z = _rand(g, 1, N, N, 128)
    mask = torch.ones((1, N, N), device="cuda", dtype=BF)
    assert m._pair_track(z, mask) is None              # not packed yet
    ref = m.pair_update(z, mask)
    assert m._pair_track(z, mask) is not None
    seen = []
    handle = m.tri_att_end.register_forward_hook(lambda mod, args, out: seen.append(1))
    assert m._pair_track(z, mask) is None and torch.equal(m.pair_update(z, mask), ref) and seen == [1]
    handle.remove()
    whole = torch.nn.modules.module.register_module_forward_hook(lambda mod, args, out: None)
    assert m._pair_track(z, mask) is None
    whole.remove()
    old = m.tri_mul_in.forward
    m.tri_mul_in.forward = lambda *a, **k: old(*a, **k)
    assert m._pair_track(z, mask) is None and torch.equal(m.pair_update(z, mask), ref)
    del m.tri_mul_in.forward
    for other in (mask.float(), mask.bool(), torch.ones((1, N, 2 * N), device="cuda", dtype=BF)[:, :, ::2]):
        assert m._pair_track(z, other) is None and torch.equal(m.pair_update(z, other), ref)
    wide = torch.zeros((1, N, N + 1, 128), device="cuda", dtype=BF)
    wide[:, :, :N] = z
    assert m._pair_track(wide[:, :, :N], mask) is None and torch.equal(m.pair_update(wide[:, :, :N], mask), ref)
    assert m._pair_track(z.float(), None) is None and m._pair_track(torch.cat([z, z]), None) is None
    ws = m.tri_mul_out._workspace
    ws["row_block"] = 16
    assert m._pair_track(z, mask) is None
    del ws["row_block"]
    m.transition_z.set_impl("reference")
    assert m._pair_track(z, mask) is None
    pairformer.set_impl(m, "fused")
    assert m._pair_track(z, mask) is None and torch.equal(m.pair_update(z, mask), ref)
    assert m._pair_track(z, mask) is not None
