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


class _OnGpu(torch.Tensor):
    """A tensor of the CPU that says it is on a GPU, so that the forms for one are chosen."""
    is_cuda = property(lambda self: True)


def _gpu(*shape, dtype=BF):
    return torch.zeros(shape, dtype=dtype).as_subclass(_OnGpu)


def _apb_weights(c, heads):
    r = lambda *s: torch.randn(s)  # noqa: E731
    return pair.ApbPacked.pack(r(c, c), r(c), r(c, c), r(c, c), r(c, c), r(c, c), heads)


@pytest.mark.parametrize("c", [376, 392, 768])
def test_attention_rows_of_another_width_are_refused(launches, c):
    planes = torch.zeros(16, 8, 8, dtype=BF)
    with pytest.raises(ValueError):
        pair.apb_fused(_gpu(1, 8, c), _apb_weights(384, 16), planes, 8)
    assert not launches
    pair.apb_fused(_gpu(1, 8, 384), _apb_weights(384, 16), planes, 8)
    assert _names(launches) == ["ubm_apb"]


def test_an_output_projection_of_another_width_is_refused(launches):
    w = _apb_weights(384, 16)
    w.wo = w.wo[:, :-32].contiguous()
    with pytest.raises(ValueError):
        pair.apb_fused(_gpu(1, 8, 384), w, torch.zeros(16, 8, 8, dtype=BF), 8)
    assert "ubm_apb" not in _names(launches)


@pytest.mark.parametrize("w12,w3,residual", [((512, 72), (64, 256), True), ((512, 56), (64, 256), True), ((256, 64), (64, 256), True),
                                             ((576, 64), (64, 256), True), ((512, 64), (32, 256), True)])
def test_transition_weights_of_another_size_are_refused(launches, w12, w3, residual):
    x = torch.zeros(9, 64, dtype=BF)
    with pytest.raises(ValueError):
        pair.transition_rows(x, None, None, 1e-5, torch.zeros(w12, dtype=BF), torch.zeros(w3, dtype=BF), residual)
    with pytest.raises(ValueError):
        pair.transition_rows(x.float(), None, None, 1e-5, torch.zeros(512, 64, dtype=BF), torch.zeros(64, 256, dtype=BF), True)
    assert not launches
    pair.transition_rows(x, None, None, 1e-5, torch.zeros(512, 64, dtype=BF), torch.zeros(64, 256, dtype=BF), True)
    assert _names(launches) == ["ubm_transition_rows"]


@pytest.mark.parametrize("c", [64, 256])
def test_atom_weights_of_another_width_are_refused(launches, c):
    """Rows of 128 channels with weights packed for others: the projections one by one say so."""
    from uplifting_biomolecular_modeling_b200.ops import atom
    r = lambda *s: torch.randn(s)  # noqa: E731
    a, rows = _gpu(1, 64, 128), _gpu(64, 128)
    w = pair.ApbPacked.pack(r(128, c), r(128), r(128, c), r(128, c), r(128, c), r(128, 128), 4)
    with pytest.raises(ValueError):
        atom.attention(a, rows, rows, w, _gpu(1, 4, 2, 32, 128), rows)
    with pytest.raises(ValueError):
        atom.transition(_gpu(1, 256, 128), _gpu(256, 128), _gpu(256, 128), _gpu(256, 128), _gpu(768, c), _gpu(128, 256))
    assert set(_names(launches)) <= {"ubm_adaln_rows"}
    atom.attention(a, rows, rows, _apb_weights(128, 4), _gpu(1, 4, 2, 32, 128), rows)
    atom.transition(_gpu(1, 256, 128), _gpu(256, 128), _gpu(256, 128), _gpu(256, 128), _gpu(768, 128), _gpu(128, 256))
    assert _names(launches)[-3:] == ["ubm_atom_qkvg", "ubm_window_layer", "ubm_cond_transition"]


@pytest.mark.parametrize("workspace", [{}, {"row_block": 16}])
@pytest.mark.parametrize("shape", [(20, 20), (1, 20), (20, 1), (1, 1), (20,), (400,), (1, 20, 20)])
def test_masks_of_a_triangle_multiplication_cover_it(monkeypatch, launches, workspace, shape):
    """What stands where the kernel will read N * N values."""
    import ctypes
    N, seen = 20, []

    class Reader:
        def __getattr__(self, name):
            def call(*args):
                if name in ("ubm_trimul", "ubm_trimul_proj"):
                    at = pair._TRIMUL_ARGS.unpack(args[0])[1] if name == "ubm_trimul" else args[4]
                    seen.append(torch.frombuffer(bytearray(ctypes.string_at(at, 4 * N * N)), dtype=torch.float32).view(N, N))
                return 0
            return call

    monkeypatch.setattr(native, "lib", lambda: Reader())
    mask = torch.rand(shape)
    pair.trimul_fused(torch.zeros(N, N, 128, dtype=BF), mask, _trimul_weights(), True, workspace=dict(workspace))
    assert len(seen) == 1 and torch.equal(seen[0], mask.reshape(N, N) if mask.numel() == N * N else mask.expand(N, N))


@pytest.mark.parametrize("workspace", [{}, {"row_block": 16}])
@pytest.mark.parametrize("shape", [(19, 20), (19, 19), (20, 21), (399,), (2, 20, 20)])
def test_masks_of_another_size_are_refused(launches, workspace, shape):
    with pytest.raises(RuntimeError):
        pair.trimul_fused(torch.zeros(20, 20, 128, dtype=BF), torch.zeros(shape), _trimul_weights(), True, workspace=dict(workspace))
    assert not launches
