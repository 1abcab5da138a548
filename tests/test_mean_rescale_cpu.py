"""Operands that the in-place rescaling of a mean refuses before anything is launched."""
import pytest
import torch

from uplifting_biomolecular_modeling_b200.ops import native, rows


@pytest.mark.parametrize("rows_,count,bias", [((3, 8), (3,), (8,)), ((3, 8), (2,), (8,)), ((3, 8), (3,), (7,))])
def test_refused_on_the_host(monkeypatch, rows_, count, bias):
    monkeypatch.setattr(native, "lib", lambda: pytest.fail("launched"))
    with pytest.raises(ValueError):
        rows.mean_rescale_(torch.zeros(rows_, dtype=torch.bfloat16), torch.ones(count), torch.zeros(bias), 2)
