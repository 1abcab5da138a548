"""Decode projections on matrix instructions: edges of the 16-row tiles and of the 64-wide blocks, every number of decode rows,
and the weights the form does not take."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _inputs(M, N, K, dual, gamma, seed, offset=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731

    def weight():
        flat = torch.empty(N * K + offset, device="cuda", dtype=torch.bfloat16)
        w = flat[offset:].view(N, K)
        return w.copy_(r(N, K) * K ** -0.5)
    return (r(M, K).bfloat16(), weight(), weight() if dual else None, 1 + 0.1 * r(K) if gamma else None, r(N),
            r(M, N).bfloat16())


def _want(x, w, w2, gamma, b, res):
    xd = x.double()
    if gamma is not None:
        xd = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-6) * gamma.double()
    y = xd @ w.double().T
    y = y + b.double() if w2 is None else F.silu(y) * (xd @ w2.double().T)
    return y + res.double()


@pytest.mark.parametrize("M", range(1, 9))
@pytest.mark.parametrize("N,K", [(1, 64), (15, 128), (17, 576), (4752, 1024)])
@pytest.mark.parametrize("dual,gamma", [(False, False), (False, True), (True, False), (True, True)])
def test_gemv_tiles(M, N, K, dual, gamma):
    from uplifting_biomolecular_modeling_b200.ops import seq
    x, w, w2, gm, b, res = _inputs(M, N, K, dual, gamma, M + N + K)
    got = seq.gemv_rows(x, w, None if dual else b, gamma=gm, w2=w2, res=res)
    want = _want(x, w, w2, gm, b, res)
    # x^ (where normalised), both halves of the SwiGLU, the projection and the sum are rounded to bf16: up to half a unit of
    # the last of 8 bits of their value each, the first two of them of the product, which the residual may cancel
    scale = want.abs() + (want - res.double()).abs() + res.double().abs()
    assert ((got.double() - want).abs() <= 5 * 2.0 ** -8 * scale + 2e-2).all()
    assert (got.double() - want).norm() <= 5 * 2.0 ** -8 * (want.norm() + (want - res.double()).norm())
    assert torch.equal(got, seq.gemv_rows(x, w, None if dual else b, gamma=gm, w2=w2, res=res))


@pytest.mark.parametrize("K,offset", [(72, 0), (128, 8)])
def test_gemv_of_other_weights(K, offset):
    """Rows that are no multiple of 64 long, and weights on 16 bytes only."""
    from uplifting_biomolecular_modeling_b200.ops import seq
    for M in (1, 5):
        x, w, _, _, b, res = _inputs(M, 33, K, False, False, K, offset)
        want = _want(x, w, None, None, b, res)
        assert (seq.gemv_rows(x, w, b, res=res).double() - want).norm() <= 3 * 2.0 ** -8 * want.norm()
