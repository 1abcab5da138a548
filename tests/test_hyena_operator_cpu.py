"""What the convolution operators of the genomic decoder keep, and which kernel a call goes to."""
import pytest
import torch

from uplifting_biomolecular_modeling_b200.models import evo2


def _operator(kind, d=16):
    cfg = evo2.replace(evo2.CONFIGS["evo2_7b"], d_model=d, n_heads=1, ffn=32)
    return evo2.HyenaOperator(cfg, kind).eval().requires_grad_(False)


def test_kept_poles_follow_the_parameter():
    op = _operator("hcl")
    exact = lambda: torch.exp(op.log_poles.float())  # noqa: E731
    assert torch.equal(op._lam(), exact())
    assert op._lam() is op._lam()
    op.log_poles.mul_(0.5)                                   # a new version
    assert torch.equal(op._lam(), exact())
    op.log_poles.data = op.log_poles.data * 0.5              # other storage, the same version
    assert torch.equal(op._lam(), exact())
    op.log_poles.data = op.log_poles.data[4:8].clone()       # a shard
    assert op._lam().shape == (4, op.cfg.state_dim) and torch.equal(op._lam(), exact())
    op.bfloat16()
    assert torch.equal(op._lam(), exact())
