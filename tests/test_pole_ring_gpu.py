"""Long convolution operator: chunks and channel blocks that are no whole number of the ring's stages, with and without 16-byte
rows, against the recurrence in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,L,d", [(1, 1, 8), (2, 15, 136), (1, 17, 12), (1, 33, 130), (2, 200, 257), (1, 1025, 264)])
@pytest.mark.parametrize("S", [1, 3, 8, 16])
@pytest.mark.parametrize("gated", [True, False])
def test_recurrence(B, L, d, S, gated):
    from uplifting_biomolecular_modeling_b200.ops import seq
    g = torch.Generator(device="cuda").manual_seed(B + L + d + S)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    u, x2 = r(B, L, d).bfloat16(), r(B, L, d).bfloat16() if gated else None
    lam, res, D = torch.rand(d, S, device="cuda", generator=g) * 0.98, r(d, S) / S, r(d)
    got, state = seq.pole_conv_gate(u, lam, res, D, x2)
    st, y = torch.zeros(B, d, S, device="cuda", dtype=torch.float64), []
    for t in range(L):
        st = st * lam.double() + u[:, t, :, None].double()
        y.append((st * res.double()).sum(-1) + D.double() * u[:, t].double())
    want = torch.stack(y, 1)
    if gated:
        want = want * x2.double()
    # fp32 recurrence; convolution, sum and product are rounded to bf16, the first before the skip term may cancel it
    assert (got.double() - want).norm() <= 4 * 2.0 ** -8 * want.norm() + 1e-3
    assert (state.double() - st).norm() <= 1e-5 * st.norm()
