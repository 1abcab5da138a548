"""Norm, projections and mask of the outer product mean in one kernel: the values of the three separate ones, rows around the edges of a
warp's 32 and of the resident grid."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("affine", [True, False])
@pytest.mark.parametrize("masked", [True, False])
@pytest.mark.parametrize("R", [1, 31, 32, 33, 127, 1000, 75776, 75809, 200003])
def test_rows(R, masked, affine):
    from uplifting_biomolecular_modeling_b200.ops import rows
    g = torch.Generator(device="cuda").manual_seed(R)
    rand = lambda *s: torch.randn(s, device="cuda", generator=g)  # noqa: E731
    m = (rand(R, 64) * 2 + 0.5).to(BF)
    ln_w, ln_b = (1 + 0.1 * rand(64), 0.1 * rand(64)) if affine else (None, None)
    wa, wb = (rand(32, 64) / 8).to(BF), (rand(64, 32) / 8).to(BF).t()             # one of them with other strides
    mask = (rand(R) > 0).to(BF) * 0.75 if masked else None
    out = rows.outer_projections(m, ln_w, ln_b, 1e-5, wa, wb, mask)
    n = rows.layernorm_rows(m, ln_w, ln_b, 1e-5)                                   # bf16, as the kernel rounds it
    for got, w in zip(out, (wa, wb)):
        ref = n.double() @ w.double().t()
        if masked:
            ref = ref * mask.double()[:, None]
        # the sum is rounded to bf16 once, and once more by the mask: 2^-8 of the value each (8 significant bits); fp32 sums of 64 terms
        # of up to a half
        assert ((got.double() - ref).abs() <= (2.01 if masked else 1.0) * 2.0 ** -8 * ref.abs() + 4e-6).all()


def test_masks_and_layouts_of_the_operator():
    """Masks of other types, strided ones, and an input that is not on 16 bytes: the same result."""
    from uplifting_biomolecular_modeling_b200.models import msa, pairformer
    torch.manual_seed(0)
    op = msa.OuterProductMean().cuda().to(BF).requires_grad_(False)
    pairformer.set_impl(op, "fused")
    S, N = 9, 40
    g = torch.Generator(device="cuda").manual_seed(2)
    m = torch.randn(1, S, N, 64, device="cuda", generator=g).to(BF)
    mask = torch.rand(1, S, N, device="cuda", generator=g) < 0.8
    ref = op(m, mask)
    wide = torch.zeros(1, S, 2 * N, device="cuda", dtype=BF)
    wide[..., ::2] = mask.to(BF)
    off = torch.empty(m.numel() + 1, device="cuda", dtype=BF)[1:].view(m.shape).copy_(m)
    assert off.data_ptr() % 16
    for x, k in ((m, mask.float()), (m, mask.to(BF)), (m, wide[..., ::2]), (off, mask)):
        assert torch.allclose(op(x, k).float(), ref.float(), rtol=2.0 ** -7, atol=1e-3)
    # one row for all sequences masks them all and counts once
    row, bias = mask[:, :1], op.proj_o.bias.float()
    once = (op(m, row.expand(1, S, N).contiguous()).float() - bias) * S + bias
    assert torch.allclose(op(m, row).float(), once, rtol=2.0 ** -6, atol=S * 2.0 ** -8)
    full = torch.ones(1, S, N, device="cuda", dtype=BF)
    part = op(m, full)
    op.full_mask = True
    assert torch.allclose(op(m, full).float(), part.float(), rtol=2.0 ** -7, atol=1e-3)
    with pytest.raises((RuntimeError, ValueError)):
        op.full_mask = False
        op(m, mask[:, :, :7])


def test_refused():
    from uplifting_biomolecular_modeling_b200.ops import rows
    m, w = torch.zeros(8, 64, device="cuda", dtype=BF), torch.zeros(32, 64, device="cuda", dtype=BF)
    for bad in ((m.float(), w, w, None), (m[:, :32], w, w, None), (m, w.float(), w, None), (m, w, w[:8], None),
                (m, w, w, torch.ones(7, device="cuda", dtype=BF)), (m, w, w, torch.ones(8, device="cuda"))):
        with pytest.raises(ValueError):
            rows.outer_projections(bad[0], None, None, 1e-5, *bad[1:])
