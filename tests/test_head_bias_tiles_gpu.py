"""Head biases whose tiles span several rows of the pair tensor, and sizes with more tiles than resident blocks (each takes several)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("N,H", [(1, 8), (3, 4), (11, 16), (127, 8), (129, 32), (275, 8), (276, 16), (401, 4), (402, 32), (640, 8)])
def test_tiles_and_rows(N, H, transpose):
    from uplifting_biomolecular_modeling_b200.ops import rows
    g = torch.Generator(device="cuda").manual_seed(N + H)
    z = torch.randn(N, N, 128, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(H, 128, device="cuda", generator=g) * 128 ** -0.5
    gamma, beta = torch.rand(128, device="cuda", generator=g) + 0.5, torch.randn(128, device="cuda", generator=g)
    planes = torch.full((H + 1, N, (N + 7) // 8 * 8), 7.0, device="cuda", dtype=torch.bfloat16)
    out = rows.pair_head_bias(z, gamma, beta, w, transpose=transpose, out=planes)
    n = torch.nn.functional.layer_norm(z.double(), (128,), gamma.double(), beta.double(), 1e-5)
    ref = torch.einsum("ijc,hc->hji" if transpose else "ijc,hc->hij", n, w.double())
    # one rounding to bf16 (2^-8 of the value) of fp32 sums of 128 terms of about one, the mean taken off behind them
    assert ((out[:H].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all()
    assert (planes[H] == 7).all() and (planes[:, :, N:] == 7).all()            # nothing beside its planes
