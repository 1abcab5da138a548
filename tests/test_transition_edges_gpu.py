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


def _weights(seed, hidden):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    return r, (1 + 0.1 * r(128), 0.1 * r(128), r(hidden, 128) / 128 ** 0.5, r(hidden, 128) / 128 ** 0.5, r(128, hidden) / hidden ** 0.5)


@pytest.mark.parametrize("hidden", [64, 512])
@pytest.mark.parametrize("ratio", [1, 100])
@pytest.mark.parametrize("shift", [0, 8])
def test_rows_far_from_zero(ratio, hidden, shift):
    """Mean and bias enter the first product as three bf16 parts each.  With a mean of 100 deviations and weights that sum up to
    1024, a mean without its last part (2^-17) would be off by 0.8 deviations, without its second by 400."""
    from uplifting_biomolecular_modeling_b200.ops import native, pair
    r, (nw, nb, a, b, o) = _weights(ratio + hidden, hidden)
    sign = torch.sign(r(3000, 64))
    x = (2.0 ** r(3000, 1).round() * (0.73 * ratio + torch.cat([sign, -sign], 1))).bfloat16()
    packed = pair.TransitionPacked.pack(nw * 0 + 1, 4 * nb, a + shift, b + shift, o)
    got = pair.transition_fused(x, packed, residual=False)
    native.raise_on_status("cuda", "transition")
    # float64 on the kernel's own folded weights: their rounding is not what is tested
    xd = x.double()
    mu, rstd = xd.mean(-1, keepdim=True), (xd.var(-1, unbiased=False, keepdim=True) + 1e-5).rsqrt()
    ab = (rstd * (xd @ packed.wab.double().T - mu * packed.colsum.double()) + packed.colbias.double()).view(len(x), -1, 2, 64)
    h = torch.nn.functional.silu(ab[:, :, 0]) * ab[:, :, 1]
    want = h.reshape(len(x), -1) @ packed.wo.double().T
    # two roundings to bf16 and tanh.approx; fp32 sums that come to mean x column sum and cancel, to 2^-24 of that a few times,
    # in both factors of values of order one; the variance as a difference of squares near (mean / deviation)^2
    size = xd.abs().amax(-1, keepdim=True) * rstd
    bound = 2.5 * 2.0 ** -9 + 2.0 ** -24 * (16 * size * packed.colsum.abs().max() + 32 * size ** 2)
    err = (got.double() - want).norm(dim=1, keepdim=True) / want.norm(dim=1, keepdim=True)
    assert (err <= bound).all(), (err / bound).max()


def test_rows_whose_squares_overflow():
    """Such a row has no variance in fp32; as in the tensor statements what is left of its norm is the bias."""
    from uplifting_biomolecular_modeling_b200.ops import native, pair
    r, (nw, nb, a, b, o) = _weights(7, 256)
    x = torch.sign(r(300, 128)).bfloat16()
    x[:, 64:] = -x[:, :64]                                       # mean 0
    x[5], x[17], x[200:232] = x[5] * 1e19, x[17] * 3e25, x[200:232] * 1e30
    x[60], x[299] = float("nan"), float("inf")
    got = pair.transition_fused(x, pair.TransitionPacked.pack(nw, nb, a, b, o), residual=False)
    native.raise_on_status("cuda", "transition")
    bias = (torch.nn.functional.silu(a.double() @ nb.double()) * (b.double() @ nb.double())) @ o.double().T
    both = pair.transition_fused(x, pair.TransitionPacked.pack(nw, nb, a, b, o), residual=True)
    rows = [5, 17, *range(200, 232)]
    assert torch.equal(both[rows], x[rows])                      # the residual dwarfs the bias
    assert ((got[rows].double() - bias).norm(dim=1) <= 5 * 2.0 ** -8 * bias.norm()).all()
    assert got[[60, 299]].isnan().all()
    rest = [i for i in range(300) if i not in rows + [60, 299]]
    want = R.transition(x[rest].double(), *(t.double() for t in (nw, nb, a, b, o)), residual=False)
    assert (got[rest].double() - want).norm() <= 5 * 2.0 ** -8 * want.norm()
