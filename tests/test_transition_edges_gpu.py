"""Pair transition at the edges of its tiles: row counts around one tile, an odd number of hidden chunks and the most it takes."""
import pytest
import torch

from uplifting_biomolecular_modeling_b200.ops import reference as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 40000])
@pytest.mark.parametrize("hidden", [192, 1024])
@pytest.mark.parametrize("residual", [False, True])
def test_transition(rows, hidden, residual):
    from uplifting_biomolecular_modeling_b200.ops import native, pair
    g = torch.Generator(device="cuda").manual_seed(rows + hidden)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    x = (r(rows, 128) * 1.5 + 0.2).bfloat16()
    nw, nb = 1 + 0.1 * r(128), 0.1 * r(128)
    a, b, o = r(hidden, 128) / 128 ** 0.5, r(hidden, 128) / 128 ** 0.5, r(128, hidden) / hidden ** 0.5
    w = pair.TransitionPacked.pack(nw, nb, a, b, o)
    keep = x.clone()
    got = pair.transition_fused(x, w, residual=residual)
    native.raise_on_status("cuda", "transition")
    assert torch.equal(x, keep)
    want = R.transition(x.double(), *(t.double() for t in (nw, nb, a, b, o)), residual=residual)
    # three weight matrices, the gated hidden values and the result are rounded to bf16 (2^-8 of their value each)
    assert (got.double() - want).norm() <= 5 * 2.0 ** -8 * want.norm()
    in_place = pair.transition_fused(x, w, residual=residual, out=x)
    assert torch.equal(in_place, got)


@pytest.mark.parametrize("hidden", [64, 128])
def test_fewest_chunks_with_several_tiles_per_cta(hidden):
    """The fewest hidden chunks against row tiles that follow one another in a CTA (four each, the last one ragged)."""
    from uplifting_biomolecular_modeling_b200.ops import native, pair
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = 3 * 128 * sms + 128 * 5 + 7
    g = torch.Generator(device="cuda").manual_seed(hidden)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    x = (r(rows, 128) * 1.5 + 0.2).bfloat16()
    nw, nb = 1 + 0.1 * r(128), 0.1 * r(128)
    a, b, o = r(hidden, 128) / 128 ** 0.5, r(hidden, 128) / 128 ** 0.5, r(128, hidden) / hidden ** 0.5
    got = pair.transition_fused(x, pair.TransitionPacked.pack(nw, nb, a, b, o), residual=True)
    native.raise_on_status("cuda", "transition")
    want = R.transition(x.double(), *(t.double() for t in (nw, nb, a, b, o)), residual=True)
    assert (got.double() - want).norm() <= 5 * 2.0 ** -8 * want.norm()
    far = (got.double() - want).norm(dim=1) > 0.1 * want.norm(dim=1)        # no tile left out
    assert not far.any()
