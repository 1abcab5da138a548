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
