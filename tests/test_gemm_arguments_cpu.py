"""Shapes that the GEMM entry point refuses or accepts, with the launch replaced by a recorder: no kernel is needed to
see which addresses one would have used."""
import pytest
import torch

from uplifting_biomolecular_modeling_b200.ops import gemm as G
from uplifting_biomolecular_modeling_b200.ops import native


@pytest.fixture
def launches(monkeypatch):
    seen = []

    class Recorder:
        @staticmethod
        def ubm_gemm_bf16_packed(args):
            f = G._ARGS.unpack(args)
            seen.append(dict(zip(("M", "N", "K", "batch", "lda", "ldb", "ldc", "ldr", "sa", "sb", "sc", "sr"), f[5:17])))
            return 0

    monkeypatch.setattr(native, "lib", lambda: Recorder)
    monkeypatch.setattr(native, "status_tensor", lambda device: torch.zeros(4, dtype=torch.int32))
    monkeypatch.setattr(native, "current_stream", lambda device=None: 0)
    return seen


def _bf(*shape):
    return torch.zeros(shape, dtype=torch.bfloat16)


@pytest.mark.parametrize("a,b", [((2, 3, 64, 128), (256, 128)), ((2, 3, 64, 128), (2, 3, 256, 128)), ((64,), (256, 64)),
                                 ((64, 128), (128,)), ((2, 64, 128), (256, 128)), ((2, 64, 128), (3, 256, 128)),
                                 ((64, 128), (256, 64))])
def test_operands_of_other_shapes_are_refused(launches, a, b):
    with pytest.raises(ValueError):
        G.gemm(_bf(*a), _bf(*b))
    assert not launches


@pytest.mark.parametrize("batch,shape", [(1, (256,)), (1, (63, 256)), (1, (64, 255)), (1, (1, 1, 64, 256)), (1, (2, 32, 255)),
                                         (1, (2, 31, 256)), (2, (128, 256)), (2, (1, 64, 256)), (2, (2, 63, 256)),
                                         (2, (2, 64, 128))])
@pytest.mark.parametrize("name", ["out", "residual"])
def test_an_output_or_residual_that_does_not_hold_the_product_is_refused(launches, batch, shape, name):
    a, b = (_bf(64, 128), _bf(256, 128)) if batch == 1 else (_bf(2, 64, 128), _bf(2, 256, 128))
    with pytest.raises(ValueError):
        G.gemm(a, b, **{name: _bf(*shape)})
    assert not launches


def test_short_output_of_a_gated_product_is_refused(launches):
    for shape in ((128,), (63, 128), (64, 256)):
        with pytest.raises(ValueError):
            G.gemm(_bf(64, 128), _bf(256, 128), act="swiglu", out=_bf(*shape))
    assert not launches


def test_forms_that_are_taken(launches):
    a, b = _bf(64, 128), _bf(256, 128)
    assert G.gemm(a, b).shape == (64, 256)
    assert G.gemm(a[None], b[None]).shape == (1, 64, 256)
    assert G.gemm(a[None], b).shape == (1, 64, 256)
    wide = _bf(70, 264)
    assert G.gemm(a, b, out=wide[:, :256], residual=wide[3:, 8:]) .shape == (70, 256)
    assert (launches[-1]["ldc"], launches[-1]["ldr"]) == (264, 264)
    G.gemm(a, b, residual=_bf(2, 32, 256))                       # rows of several entries back to back
    G.gemm(a, b, residual=_bf(1, 256).expand(64, 256))           # one row for all
    assert launches[-1]["ldr"] == 0
    three = _bf(3, 80, 256)
    assert G.gemm(_bf(3, 64, 128), _bf(3, 256, 128), out=three, residual=three).shape == (3, 80, 256)
    assert [launches[-1][k] for k in ("batch", "ldc", "sc", "ldr", "sr")] == [3, 256, 80 * 256, 256, 80 * 256]
    assert G.gemm(_bf(128, 64), _bf(128, 256), mn_major=True).shape == (64, 256)
    assert launches[-1]["M"] == 64 and launches[-1]["K"] == 128
