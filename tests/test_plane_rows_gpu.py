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


@pytest.mark.parametrize("N", [9, 129])
def test_projection_statistics(N):
    """Row means of the projection as the sum of four parts of 32 channels: results do not depend on which warp takes them."""
    from uplifting_biomolecular_modeling_b200.ops import native, pair
    g = torch.Generator(device="cuda").manual_seed(N)
    c = 128
    z = (_rand((N, N, c), g, 3.0) + 40.0).bfloat16()
    one, zero = torch.ones(c, device="cuda"), torch.zeros(c, device="cuda")
    w = pair.TrimulPacked.pack(one, zero, *(_rand((2 * c, c), g) for _ in range(2)), one, zero, *(_rand((c, c), g) for _ in range(2)))
    Np = pair.ceil_to(N, pair.PLANE_ROW)
    planes = torch.empty(2, 128, N, Np, device="cuda", dtype=torch.bfloat16)
    stats = torch.empty(N * N, 2, device="cuda")
    rc = native.lib().ubm_trimul_proj(native.ptr(z), native.ptr(w.w_in), native.ptr(w.in_colsum), native.ptr(w.in_colbias), 0,
                                      native.ptr(planes), native.ptr(stats), N, Np, native.ptr(native.status_tensor(z.device)),
                                      native.current_stream(z.device))
    native.check(rc, "ubm_trimul_proj")
    native.raise_on_status("cuda", "trimul_proj")
    x = z.float().view(N * N, 4, 16, 2)
    pairs, part = x[..., 0] + x[..., 1], torch.zeros(N * N, 4, device="cuda")
    for k in range(16):
        part = part + pairs[:, :, k]
    mean = ((part[:, 0] + part[:, 1]) + (part[:, 2] + part[:, 3])) / 128
    assert torch.equal(stats[:, 0], mean)
    var = z.double().view(N * N, c).var(-1, unbiased=False)
    # single-pass variance: fp32 sums of squares near 40^2 + 3^2 (2^-24 of 1609 for each of about 40 roundings) against 9
    assert ((stats[:, 1].double() * (var + 1e-5).sqrt() - 1).abs() <= 40 * 2 ** -24 * 1609 / 9).all()


@pytest.mark.parametrize("row", [8, 16])
@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("H", [4, 16])
@pytest.mark.parametrize("N", [7, 8, 24, 33, 48, 129])
def test_head_bias_padding(monkeypatch, N, H, transpose, row):
    """Planes of its own have zeros behind every row, whatever the memory held; planes given to it keep their rows' length and what
    lies behind column N."""
    from uplifting_biomolecular_modeling_b200.ops import rows
    g = torch.Generator(device="cuda").manual_seed(N + H)
    z, w = _rand((N, N, 128), g).bfloat16(), _rand((H, 128), g, 128 ** -0.5)
    one, zero = torch.ones(128, device="cuda"), torch.zeros(128, device="cuda")
    Np = (N + row - 1) // row * row
    real = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, **k: real(*a, **k).fill_(float("nan")))
    own = rows.pair_head_bias(z, one, zero, w, transpose=transpose, row=row)
    monkeypatch.undo()
    whole = own.as_strided((H, N, Np), (N * Np, Np, 1))
    assert own.stride() == (N * Np, Np, 1) and not whole[:, :, N:].any() and own.isfinite().all()
    for ld in {(N + 7) // 8 * 8, Np, Np + 8}:
        planes = torch.full((H, N, ld), 5.0, device="cuda", dtype=torch.bfloat16)
        for given in (planes, planes[:, :, :N]):
            planes[:, :, :N] = 5.0
            got = rows.pair_head_bias(z, one, zero, w, transpose=transpose, out=given)
            assert torch.equal(got, own) and torch.equal(planes[:, :, :N], own) and (planes[:, :, N:] == 5).all()


def test_head_bias_planes_that_do_not_fit():
    from uplifting_biomolecular_modeling_b200.ops import rows
    z, w = torch.zeros(24, 24, 128, device="cuda", dtype=torch.bfloat16), torch.zeros(4, 128, device="cuda")
    planes = torch.zeros(4, 24, 32, device="cuda", dtype=torch.bfloat16)
    for out in (planes.float(), planes[:3], planes[:, :23], planes[:, :, :23], planes.cpu(), planes[:, ::2], planes.view(4, -1),
                torch.zeros(4, 24, 28, device="cuda", dtype=torch.bfloat16), torch.zeros(4, 25, 24, device="cuda", dtype=torch.bfloat16)):
        with pytest.raises(ValueError):
            rows.pair_head_bias(z, None, None, w, out=out)


@pytest.mark.parametrize("N", [24, 33])
def test_attention_asks_for_rows_of_eight(N):
    """Padding to sectors would cost the planes of 24 tokens a fill and gain the attention nothing."""
    from uplifting_biomolecular_modeling_b200.models import pairformer
    with torch.device("cuda"):
        m = pairformer.AttentionPairBias().bfloat16().eval().requires_grad_(False)
    pairformer.set_impl(m, "fused")
    planes = m.pair_bias(torch.zeros(1, N, N, 128, device="cuda", dtype=torch.bfloat16))
    assert planes.ld == (N + 7) // 8 * 8
