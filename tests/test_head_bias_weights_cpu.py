"""The folded weights of the pair head biases: kept from call to call, and made anew when any of the parameters behind them changes."""
import pytest
import torch

from uplifting_biomolecular_modeling_b200.ops import rows


def _params():
    torch.manual_seed(3)
    return [torch.nn.Parameter(torch.randn(s)) for s in ((4, 128), (128,), (128,))]


def _reference(w, g, b, scale):
    w64, g64, b64 = (t.detach().double() for t in (w, g, b))
    wf = w64 * g64 * scale
    return wf, wf.sum(1), w64 @ b64 * scale


def _check(p, scale=1.5):
    # fp32 sums of 128 products: 128 roundings of 2^-24 of a sum of magnitudes below 128 * 16
    for got, ref in zip(rows._head_bias_weights(*p, scale, "cpu"), _reference(*p, scale)):
        assert (got.double() - ref).abs().max() < 128 * 2.0 ** -24 * 2048


def test_unchanged_parameters_keep_their_form():
    p = _params()
    assert all(a is b for a, b in zip(rows._head_bias_weights(*p, 1.5, "cpu"), rows._head_bias_weights(*p, 1.5, "cpu")))


@pytest.mark.parametrize("which", [0, 1, 2])
def test_a_parameter_written_in_place_counts(which):
    p = _params()
    _check(p)
    with torch.no_grad():
        p[which].mul_(2.0)
    _check(p)


@pytest.mark.parametrize("which", [0, 1, 2])
def test_another_parameter_counts(which):
    p = _params()
    _check(p)
    p[which] = torch.nn.Parameter(p[which].detach() + 1.0)       # of the same version
    _check(p)


@pytest.mark.parametrize("which", [0, 1, 2])
def test_other_storage_counts(which):
    p = _params()
    _check(p)
    p[which].data = p[which].detach() - 1.0                      # leaves the version as it is
    _check(p)


def test_a_norm_with_and_without_a_shift():
    w, g, b = _params()
    assert rows._head_bias_weights(w, g, b, 1.0, "cpu")[2].abs().max() > 0
    assert rows._head_bias_weights(w, g, None, 1.0, "cpu")[2].abs().max() == 0
    _check([w, g, b], 1.0)
