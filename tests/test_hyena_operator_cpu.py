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


class _Recorder:
    """In the library's place: remembers which entry a call went to."""

    def __init__(self):
        self.seen = []

    def __getattr__(self, name):
        return lambda *a: self.seen.append(name) or 0


@pytest.fixture
def entries(monkeypatch):
    from uplifting_biomolecular_modeling_b200.ops import native
    lib = _Recorder()
    monkeypatch.setattr(native, "lib", lambda: lib)
    monkeypatch.setattr(native, "current_stream", lambda device=None: 0)
    return lib.seen


def test_more_sequences_than_a_grid_holds(entries):
    """65536 sequences: the long operator takes the transform, the medium one the kernel that walks a flat index."""
    from uplifting_biomolecular_modeling_b200.ops import seq
    op = _operator("hcl", 8)
    for B, want in ((2, ["ubm_pole_conv_gate"]), (65536, ["ubm_fft_pad_transpose", "ubm_spectrum_mul", "ubm_fftconv_epilogue"])):
        u = torch.zeros(B, 1, 8, dtype=torch.bfloat16)
        op._fused_inner(u, u, {})
        assert entries == want
        entries.clear()
    ht, D = torch.zeros(128, 8), torch.zeros(8)
    for B, want in ((2, "ubm_fir_toeplitz"), (65536, "ubm_fir_inner_gate")):
        u = torch.zeros(B, 64, 8, dtype=torch.bfloat16)
        seq.fir_inner_gate(u, ht, D, u, taps_bf16=True)
        assert entries.pop() == want


@pytest.mark.parametrize("lam,res,D,x2", [((4, 3), (8, 3), (8,), (1, 2, 8)), ((8, 3), (8, 2), (8,), (1, 2, 8)),
                                          ((8, 3), (8, 3), (4,), (1, 2, 8)), ((8, 3), (8, 3), (8,), (1, 1, 8))])
def test_poles_of_other_channels_are_refused(entries, lam, res, D, x2):
    from uplifting_biomolecular_modeling_b200.ops import seq
    u = torch.zeros(1, 2, 8, dtype=torch.bfloat16)
    with pytest.raises(ValueError):
        seq.pole_conv_gate(u, torch.zeros(lam), torch.zeros(res), torch.zeros(D), torch.zeros(x2))
    assert not entries
