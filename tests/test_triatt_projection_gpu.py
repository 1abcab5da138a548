"""Projection of triangle attention on its own: q, k, v, the gate and the head biases at sizes around its 16-row boxes, its
128-row tiles and the 8-wide rows of the bias planes, written in place and at the transposed pair."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("starting", [True, False])
@pytest.mark.parametrize("N", [7, 15, 16, 17, 31, 33, 127, 129, 150, 200])
def test_projection_rows(N, starting):
    from uplifting_biomolecular_modeling_b200.ops import native, pair
    g = torch.Generator(device="cuda").manual_seed(N)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    c, H = 128, 4
    z = (r(N, N, c) + 0.2).bfloat16()
    ws = [r(c, c) * c ** -0.5 for _ in range(4)]
    w = pair.TriattPacked.pack(1 + 0.1 * r(c), 0.1 * r(c), r(H, c) * c ** -0.5, *ws, 0.1 * r(c), r(c, c) * c ** -0.5, r(c), H)
    space = {}
    pair.triangle_attention_fused(z, w, starting=starting, residual=False, workspace=space)
    torch.cuda.synchronize()
    native.raise_on_status("cuda", "triangle attention")
    (qkvgo, hb), = space.values()

    zd = (z if starting else z.transpose(0, 1)).double().reshape(N * N, c)
    mean, rstd = zd.mean(-1, keepdim=True), (zd.var(-1, unbiased=False, keepdim=True) + 1e-5).rsqrt()

    def project(weight, colsum, colbias):
        return rstd * (zd @ weight.double().T - mean * colsum.double()) + colbias.double()
    want = project(w.w, w.colsum, w.colbias)
    want[:, 384:] = want[:, 384:].sigmoid()
    got = torch.cat([qkvgo[i] for i in range(4)], -1).double()
    # one rounding to bf16, sums of 128 products in fp32 (values up to 5), and the gate's tanh.approx: 2^-11 of a value to 1
    assert ((got - want).abs() <= 2 ** -8 * want.abs() + 2 ** -11).all()
    wantb = project(w.wb, w.wb_colsum, w.wb_colbias).T.reshape(H, N, N)
    assert ((hb[:, :, :N].double() - wantb).abs() <= 2 ** -8 * wantb.abs() + 2 ** -11).all()
    assert not hb[:, :, N:].any()
