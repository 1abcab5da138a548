"""Triangle multiplication and head-bias planes at row lengths around the padding of a plane's rows (16 elements)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(shape, g, k=1.0):
    return torch.randn(*shape, device="cuda", generator=g) * k


@pytest.mark.parametrize("outgoing", [True, False])
@pytest.mark.parametrize("N", [8, 9, 24, 25, 40, 120, 129])
def test_trimul_rows(N, outgoing):
    from uplifting_biomolecular_modeling_b200.ops import native, pair, reference
    g = torch.Generator(device="cuda").manual_seed(N)
    c = 128
    z = (_rand((N, N, c), g) + 0.2).bfloat16()
    mask = (torch.rand((N, N), device="cuda", generator=g) > 0.1).float()
    norms = [f(_rand((c,), g, 0.1)) for f in (lambda t: 1 + t, lambda t: t)] * 2
    p_in, g_in = _rand((2 * c, c), g, c ** -0.5), _rand((2 * c, c), g, c ** -0.5)
    p_out, g_out = _rand((c, c), g, c ** -0.5), _rand((c, c), g, c ** -0.5)
    w = pair.TrimulPacked.pack(*norms[:2], p_in, g_in, *norms[2:], p_out, g_out)
    # what the buffers held before does not count: their padded columns are written or never read
    space = {}
    pair.trimul_fused(torch.full_like(z, 3.0), None, w, outgoing=outgoing, residual=False, workspace=space)
    for planes in next(iter(space.values())):
        assert planes.shape[-1] % 16 == 0
        planes.fill_(float("nan"))
    out = pair.trimul_fused(z, mask, w, outgoing=outgoing, residual=False, workspace=space)
    torch.cuda.synchronize()
    native.raise_on_status("cuda", "trimul")
    ref = reference.triangle_multiplication(z.float(), mask, *norms[:2], p_in, g_in, *norms[2:], p_out, g_out,
                                            outgoing=outgoing)
    # bf16 operands of three products in a row, each rounded to 2^-9 of its value: 2 % of the mean, 6 % of the largest
    err = (out.float() - ref).abs()
    assert err.mean().item() < 2e-2 * ref.abs().mean().item()
    assert err.max().item() < 6e-2 * ref.abs().max().item()


@pytest.mark.parametrize("N", [8, 24, 25, 33])
def test_head_bias_rows(N):
    from uplifting_biomolecular_modeling_b200.ops import rows
    g = torch.Generator(device="cuda").manual_seed(N)
    z, w = _rand((N, N, 128), g).bfloat16(), _rand((4, 128), g, 128 ** -0.5)
    one, zero = torch.ones(128, device="cuda"), torch.zeros(128, device="cuda")
    planes = rows.pair_head_bias(z, one, zero, w)
    given = torch.zeros(4, N, (N + 7) // 8 * 8, device="cuda", dtype=torch.bfloat16)
    rows.pair_head_bias(z, one, zero, w, out=given)
    assert planes.stride(1) % 16 == 0 and torch.equal(planes, given[:, :, :N])
    whole = planes.as_strided((4, N, planes.stride(1)), planes.stride())
    assert not whole[:, :, N:].any()
