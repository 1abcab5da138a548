"""The forms of a projection's weight and bias that the decoder keeps: the same ones from call to call, new ones when either changes."""
import pytest
import torch
import torch.nn as nn

from uplifting_biomolecular_modeling_b200.models import evo2


def _check(m):
    w, b = evo2._bf16_weight(m)
    q, dq, b8 = evo2._e4m3_weight(m)
    assert torch.equal(w, m.weight.detach().to(torch.bfloat16)) and torch.equal(b, m.bias.detach().float()) and torch.equal(b8, b)
    assert (q.float() * dq - m.weight.detach()).abs().max() <= m.weight.detach().abs().max() * 2.0 ** -4      # 3 bits of mantissa


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("name", ["weight", "bias"])
@pytest.mark.parametrize("change", ["in_place", "other", "storage"])
def test_what_changes_counts(dtype, name, change):
    torch.manual_seed(0)
    m = nn.Linear(32, 16).to(dtype)
    _check(m)
    kept = evo2._bf16_weight(m), evo2._e4m3_weight(m)
    assert kept[0][0] is evo2._bf16_weight(m)[0] and kept[1][0] is evo2._e4m3_weight(m)[0]
    p = getattr(m, name)
    if change == "in_place":
        with torch.no_grad():
            p.mul_(-2.0)
    elif change == "other":
        setattr(m, name, nn.Parameter(p.detach() * -2.0))
    else:
        p.data = p.detach() * -2.0
    _check(m)


def test_a_bias_that_comes_and_goes():
    m = nn.Linear(32, 16, bias=False)
    assert evo2._bf16_weight(m)[1] is None and evo2._e4m3_weight(m)[2] is None
    m.bias = nn.Parameter(torch.ones(16))
    _check(m)
    m.bias = None
    assert evo2._bf16_weight(m)[1] is None and evo2._e4m3_weight(m)[2] is None
