"""Key masks laid out on the device equal the ones laid out by tensor statements, for the strides and types a mask has."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,nk", [(1, 1), (3, 63), (40, 64), (33, 65), (137, 200)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.bool, torch.uint8, torch.int64, torch.float16])
@pytest.mark.parametrize("form", ["rows", "transposed", "expanded", "strided"])
def test_lay_out_equals_pack(rows, nk, dtype, form):
    from uplifting_biomolecular_modeling_b200.ops import pair
    g = torch.Generator(device="cuda").manual_seed(rows + nk)
    keep = (torch.rand(rows, nk, device="cuda", generator=g) < 0.97).to(dtype)
    if form == "transposed":
        keep = keep.t().contiguous().t()
    elif form == "expanded":
        keep = keep[:1].expand(rows, nk)
    elif form == "strided":
        keep = torch.stack([keep, (keep == 0).to(dtype)], -1)[..., 0]
    got, want = pair.KeyMask.lay_out(keep), pair.KeyMask.pack(keep)
    if want is None:
        assert not got.add.any() and not got.flags.any()
        return
    assert torch.equal(got.add[:, :nk], want.add[:, :nk]) and torch.equal(got.flags, want.flags)
    assert got.add.shape == want.add.shape and not got.add[:, nk:].any()


def test_a_mask_that_keeps_everything_changes_nothing():
    from uplifting_biomolecular_modeling_b200.ops import pair
    q, k, v = (torch.randn(5, 130, 128, device="cuda").bfloat16() for _ in range(3))
    outs = []
    for mask in (None, pair.KeyMask.lay_out(torch.ones(5, 130, device="cuda"))):
        out = torch.empty_like(q)
        pair.attention_d32(q, k, v, None, None, out, 5, 130, 130, 4, mask=mask)
        outs.append(out)
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bool])
def test_a_mask_on_the_host_or_of_fewer_rows(dtype):
    from uplifting_biomolecular_modeling_b200.ops import pair
    keep = (torch.rand(90, 130, generator=torch.Generator().manual_seed(1)) < 0.9).to(dtype)
    dev = torch.device("cuda", torch.cuda.current_device())
    want = pair.KeyMask.lay_out(keep.to(dev))
    got = pair.KeyMask.lay_out(keep, device=dev)
    assert got.add.device == dev and torch.equal(got.add, want.add) and torch.equal(got.flags, want.flags)
    got = pair.KeyMask.lay_out(keep[:1], (90, 130), dev)
    want = pair.KeyMask.lay_out(keep[:1].to(dev).repeat(90, 1))
    assert torch.equal(got.add, want.add) and torch.equal(got.flags, want.flags)
    with pytest.raises(ValueError):
        pair.KeyMask.lay_out(keep)


def test_triangle_attention_takes_the_mask_it_took():
    """A pair mask on the host, and one that broadcasts over the attention rows, give what the expanded mask gives."""
    from uplifting_biomolecular_modeling_b200.models import pairformer
    torch.manual_seed(0)
    n = 70
    keys = torch.ones(1, 1, n)
    keys[..., 60:] = 0
    z = torch.randn(1, n, n, 128, device="cuda").bfloat16()
    m = pairformer.TriangleAttention(starting=True).cuda().bfloat16().eval().requires_grad_(False)
    pairformer.set_impl(m, "fused")
    want = m(z, keys.expand(1, n, n).cuda().contiguous(), residual=True)
    assert torch.equal(m(z, keys.cuda(), residual=True), want)
    assert torch.equal(m(z, keys.expand(1, n, n), residual=True), want)


@pytest.mark.parametrize("rows,N,D,variant", [(1, 128, 32, 0), (3, 128, 32, 0), (5, 128, 32, 0x10), (5, 192, 64, 0x10),
                                              (3, 200, 32, 0), (5, 200, 32, 0), (5, 128, 32, 0), (5, 200, 64, 0)])
def test_a_row_without_keys_is_finite(rows, N, D, variant, request):
    """The first row keeps no key.  No key count or form gives it a NaN (which would travel on through P.V of a later
    attention over these rows); it is 0, give or take the 2^-125 that is the smallest polynomial exponential, except where
    whole key steps leave those the only weights.  The other rows do not notice it."""
    from uplifting_biomolecular_modeling_b200.ops import pair
    pair.set_attention_variant(variant)
    request.addfinalizer(lambda: pair.set_attention_variant(0))
    q, k, v = (torch.randn(rows, N, 4 * D, device="cuda").bfloat16() for _ in range(3))
    keep = torch.rand(rows, N, device="cuda") < 0.9
    outs = []
    for some in (0.0, 1.0):
        keep[0] = bool(some)
        out = torch.empty_like(q)
        pair.attention(q, k, v, None, None, out, rows, N, N, 4, D, mask=pair.KeyMask.lay_out(keep))
        outs.append(out)
    assert outs[0].isfinite().all() and torch.equal(outs[0][1:], outs[1][1:])
    poly = variant == 0 and (D == 64 or rows >= 4)
    if not poly or N % 64:
        assert outs[0][0].abs().max() <= 2.0 ** -100
