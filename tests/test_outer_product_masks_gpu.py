"""Outer-product mean of sequences that cover a part of the target: token counts on and off the GEMM's alignment, masks of
several types, one mask value per sequence, pairs that no sequence covers."""
import pytest
import torch

from uplifting_biomolecular_modeling_b200.ops import reference as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,N", [(1, 8), (3, 9), (17, 64), (40, 131), (130, 136)])
@pytest.mark.parametrize("form", ["bf16", "fp32", "fractions", "per_sequence", "none"])
def test_masked_mean(S, N, form):
    from uplifting_biomolecular_modeling_b200.models import msa, pairformer
    from uplifting_biomolecular_modeling_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(S + N)
    with torch.device("cuda"):
        m = msa.OuterProductMean()
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(torch.randn(p.shape, device="cuda", generator=g) / max(1, p.shape[-1]) ** 0.5)
    m = m.bfloat16().eval().requires_grad_(False)
    pairformer.set_impl(m, "fused")
    x = torch.randn(1, S, N, 64, device="cuda", generator=g).bfloat16()
    keep = (torch.rand(1, S, N, device="cuda", generator=g) < 0.6).float()
    mask = {"bf16": keep.bfloat16(), "fp32": keep, "fractions": (keep * 0.3).bfloat16(), "none": keep.bfloat16() * 0,
            "per_sequence": keep[:, :, :1].bfloat16().expand(1, S, N)}[form]
    got = m(x, mask)
    native.raise_on_status("cuda", "outer product")
    d = lambda t: t.double()  # noqa: E731
    want = R.outer_product_mean(d(x), d(mask), d(m.norm.weight), d(m.norm.bias), d(m.proj_a.weight), d(m.proj_b.weight),
                                d(m.proj_o.weight), d(m.proj_o.bias))
    # normalised rows, projections (and their masks), the product over sequences and two roundings of the result: six of up
    # to 2^-9; the rescaled sum and the bias may cancel
    assert (d(got) - want).norm() <= 6 * 2.0 ** -9 * (want.norm() + d(m.proj_o.bias).norm() * N)


@pytest.mark.parametrize("what", ["mask", "bias"])
def test_operands_that_start_between_16_bytes(what):
    """A sequence mask, or an fp32 output bias, that is a view into a longer buffer."""
    from uplifting_biomolecular_modeling_b200.models import msa, pairformer
    from uplifting_biomolecular_modeling_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(5)
    with torch.device("cuda"):
        m = msa.OuterProductMean()
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(torch.randn(p.shape, device="cuda", generator=g) / max(1, p.shape[-1]) ** 0.5)
    m = m.bfloat16().eval().requires_grad_(False)
    pairformer.set_impl(m, "fused")
    S, N = 24, 64
    x = torch.randn(1, S, N, 64, device="cuda", generator=g).bfloat16()
    mask = (torch.rand(1, S, N, device="cuda", generator=g) < 0.6).bfloat16()
    m.proj_o.bias = torch.nn.Parameter(m.proj_o.bias.float(), requires_grad=False)
    want = m(x, mask)
    if what == "mask":
        mask = torch.empty(S * N + 1, device="cuda", dtype=torch.bfloat16)[1:].view(1, S, N).copy_(mask)
        assert mask.data_ptr() % 16
    else:
        buf = torch.empty(129, device="cuda")[1:].copy_(m.proj_o.bias)
        m.proj_o.bias = torch.nn.Parameter(buf, requires_grad=False)
        assert m.proj_o.bias.data_ptr() % 16
    got = m(x, mask)
    native.raise_on_status("cuda", "outer product")
    assert torch.equal(got, want)


@pytest.mark.parametrize("S,N", [(3, 9), (17, 64), (40, 131)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_one_row_of_the_mask_for_all_sequences(S, N, dtype):
    """The plain statements count such a row once; so does the kernel path."""
    from uplifting_biomolecular_modeling_b200.models import msa, pairformer
    from uplifting_biomolecular_modeling_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(S + N)
    with torch.device("cuda"):
        m = msa.OuterProductMean()
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(torch.randn(p.shape, device="cuda", generator=g) / max(1, p.shape[-1]) ** 0.5)
    m = m.bfloat16().eval().requires_grad_(False)
    pairformer.set_impl(m, "fused")
    x = torch.randn(1, S, N, 64, device="cuda", generator=g).bfloat16()
    mask = (torch.rand(1, 1, N, device="cuda", generator=g) < 0.6).to(dtype)
    got = m(x, mask)
    native.raise_on_status("cuda", "outer product")
    d = lambda t: t.double()  # noqa: E731
    want = R.outer_product_mean(d(x), d(mask), d(m.norm.weight), d(m.norm.bias), d(m.proj_a.weight), d(m.proj_b.weight),
                                d(m.proj_o.weight), d(m.proj_o.bias))
    # as above
    assert (d(got) - want).norm() <= 6 * 2.0 ** -9 * (want.norm() + d(m.proj_o.bias).norm() * N)
