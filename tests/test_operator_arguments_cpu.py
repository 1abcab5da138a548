"""Tensors that the operators of one call refuse or accept, with the launches replaced by a recorder: no kernel is needed to see which
addresses one would have used."""
import pytest
import torch

from uplifting_biomolecular_modeling_b200.ops import gemm as G
from uplifting_biomolecular_modeling_b200.ops import native, pair

BF = torch.bfloat16


@pytest.fixture
def launches(monkeypatch):
    seen = []

    class Recorder:
        def __getattr__(self, name):
            return lambda *args: seen.append((name, args)) or 0

    monkeypatch.setattr(native, "lib", lambda: Recorder())
    monkeypatch.setattr(native, "status_tensor", lambda device: torch.zeros(4, dtype=torch.int32))
    monkeypatch.setattr(native, "current_stream", lambda device=None: 0)
    return seen


def _names(launches):
    return [name for name, _ in launches]


def _triatt_weights():
    r = lambda *s: torch.randn(s)  # noqa: E731
    return pair.TriattPacked.pack(r(128), r(128), r(4, 128), r(128, 128), r(128, 128), r(128, 128), r(128, 128), None, r(128, 128), None, 4)


def _trimul_weights():
    r = lambda *s: torch.randn(s)  # noqa: E731
    return pair.TrimulPacked.pack(r(128), r(128), r(256, 128), r(256, 128), r(128), r(128), r(128, 128), r(128, 128))


def _triatt(z, out, workspace=None):
    return pair.triangle_attention_fused(z, _triatt_weights(), True, out=out, workspace=workspace)


def _trimul(z, out, workspace=None):
    return pair.trimul_fused(z, None, _trimul_weights(), True, out=out, workspace=workspace)


def _transition(z, out, workspace=None):
    r = lambda *s: torch.randn(s)  # noqa: E731
    return pair.transition_fused(z, pair.TransitionPacked.pack(r(128), r(128), r(256, 128), r(256, 128), r(128, 256)), out=out)


@pytest.mark.parametrize("call", [_triatt, _trimul, _transition])
@pytest.mark.parametrize("out", [(5, 6, 128), (5, 5, 128), (35, 128), (6, 6, 64), (6, 6, 256), (1,)])
def test_an_output_of_another_size_is_refused(launches, call, out):
    with pytest.raises((ValueError, RuntimeError)):
        call(torch.zeros(6, 6, 128, dtype=BF), torch.zeros(out, dtype=BF))
    assert not launches


@pytest.mark.parametrize("call", [_triatt, _trimul, _transition])
@pytest.mark.parametrize("out", [torch.zeros(6, 6, 128, dtype=torch.float16), torch.zeros(6, 6, 128, dtype=torch.int16),
                                 torch.zeros(6, 6, 128, dtype=BF).transpose(0, 1), torch.zeros(6, 128, 6, dtype=BF).transpose(1, 2),
                                 torch.zeros(6, 6, 128, dtype=BF, device="meta")])
def test_an_output_of_another_form_is_refused(launches, call, out):
    with pytest.raises((ValueError, RuntimeError)):
        call(torch.zeros(6, 6, 128, dtype=BF), out)
    assert not launches


@pytest.mark.parametrize("call", [_trimul, _transition])
@pytest.mark.parametrize("out", [torch.zeros(6, 6, 128), torch.zeros(6, 6, 192, dtype=BF)[:, :, :128]])
def test_outputs_that_only_a_product_writes_are_refused_by_the_others(launches, call, out):
    with pytest.raises(ValueError):
        call(torch.zeros(6, 6, 128, dtype=BF), out)
    assert not launches


@pytest.mark.parametrize("call,name", [(_triatt, "ubm_triatt"), (_trimul, "ubm_trimul"), (_transition, "ubm_transition")])
@pytest.mark.parametrize("shape", [(6, 6, 128), (36, 128), (1, 6, 6, 128)])
def test_outputs_that_are_taken(launches, call, name, shape):
    out = torch.zeros(shape, dtype=BF)
    assert call(torch.zeros(6, 6, 128, dtype=BF), out) is out
    assert _names(launches) == [name]


@pytest.mark.parametrize("out", [torch.zeros(6, 6, 128), torch.zeros(6, 6, 192, dtype=BF)[:, :, :128]])
def test_triangle_attention_writes_fp32_and_wider_rows_by_its_last_product(launches, out):
    z = torch.zeros(6, 6, 128, dtype=BF)
    assert _triatt(z, out) is out
    assert _names(launches) == ["ubm_triatt_proj", "ubm_attention_d32", "ubm_gemm_bf16_packed"]
    f = G._ARGS.unpack(launches[-1][1][0])
    assert f[2] == out.data_ptr() and f[4] == z.data_ptr() and f[5:8] == (36, 128, 128) and f[11] == out.stride(1)
    assert f[18] == (out.dtype == torch.float32)


def test_outputs_of_row_blocks_keep_their_shape(launches):
    z = torch.zeros(32, 32, 128, dtype=BF)
    for out in (torch.zeros(32 * 32, 128, dtype=BF), torch.zeros(32, 32, 192, dtype=BF)[:, :, :128], torch.zeros(32, 32, 128)):
        with pytest.raises(ValueError):
            _trimul(z, out, {"row_block": 16})
    assert not launches
    out = torch.zeros(32, 32, 128, dtype=BF)
    assert _trimul(z, out, {"row_block": 16}) is out
