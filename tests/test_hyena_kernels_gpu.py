"""Prefill kernels of the long and the medium convolution operator against float64 statements."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# conv, conv + skip and the gated product are rounded to bf16 (8 significant bits) one after the other: each adds at
# most 2^-8 of its value, which is at most 1 + 2^-8 of the exact one's
ROUNDINGS = 3 * 2.0 ** -8 * (1 + 2.0 ** -7)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _conv(u, h):
    """Causal convolution of [B, L, d] with [d, T] in float64 by shifted sums."""
    y = torch.zeros_like(u)
    for t in range(min(h.shape[1], u.shape[1])):
        y[:, t:] += u[:, :u.shape[1] - t] * h[:, t]
    return y


def _bound(y, u, D, x2):
    g = 1.0 if x2 is None else x2.double().abs()
    return ROUNDINGS * g * (y.abs() + (u.double() * D.double()).abs()) + 1e-5 * y.abs().max()


@pytest.mark.parametrize("B,L,d,S,gated", [(1, 1, 8, 16, True), (2, 31, 40, 3, True), (1, 33, 136, 8, False),
                                           (3, 1000, 72, 16, True), (1, 2500, 256, 5, True)])
def test_pole_conv_gate(B, L, d, S, gated):
    from uplifting_biomolecular_modeling_b200.ops import seq
    g = _gen(L)
    u = torch.randn(B, L, d, device="cuda", generator=g).bfloat16()
    x2 = torch.randn(B, L, d, device="cuda", generator=g).bfloat16() if gated else None
    lam = 1 - 10 ** -(torch.rand(d, S, device="cuda", generator=g) * 3.5 + 0.1)
    lam[0, 0] = 0.0                                             # 0^0 = 1: the first tap only
    res = torch.randn(d, S, device="cuda", generator=g) / S
    D = torch.randn(d, device="cuda", generator=g)
    out, state = seq.pole_conv_gate(u, lam, res, D, x2)
    pw = lam.double().unsqueeze(-1) ** torch.arange(L, device="cuda", dtype=torch.float64)
    y = _conv(u.double(), torch.einsum("cs,cst->ct", res.double(), pw))
    ref = (y + u.double() * D.double()) * (1.0 if x2 is None else x2.double())
    assert ((out.double() - ref).abs() <= _bound(y, u, D, x2)).all()
    want = torch.einsum("blc,csl->bcs", u.double(), pw.flip(-1))
    # fp32 recurrence: one rounding of the running state per position, each decaying like the state itself
    assert (state.double() - want).abs().max() <= 2.0 ** -23 * L ** 0.5 * 8 * want.abs().max()
    assert torch.equal(seq.pole_prefill_state(u, lam), state)


def test_pole_chunks_fit_a_grid_and_cover_the_sequence():
    from uplifting_biomolecular_modeling_b200.ops import seq
    for B, L, d in [(1, 1, 8), (1, 8192, 4096), (8, 8192, 4096), (1, 1 << 20, 4096), (1, 200_000_000, 8)]:
        c = seq._pole_chunk(B, L, d)
        assert 32 <= c and (L + c - 1) // c <= 65535


@pytest.mark.parametrize("K,L,d", [(65, 64, 8), (128, 64, 40), (100, 511, 72), (127, 513, 32), (128, 1300, 136)])
@pytest.mark.parametrize("gated", [True, False])
def test_medium_filter_on_the_tensor_cores(K, L, d, gated):
    from uplifting_biomolecular_modeling_b200.ops import seq
    g = _gen(K + L)
    u = torch.randn(2, L, d, device="cuda", generator=g).bfloat16()
    x2 = torch.randn(2, L, d, device="cuda", generator=g).bfloat16() if gated else None
    h = (torch.randn(d, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    D = torch.randn(d, device="cuda", generator=g)
    out = seq.fir_inner_gate(u, seq.taps_major(h), D, x2, taps_bf16=True)
    y = _conv(u.double(), h.double())
    ref = (y + u.double() * D.double()) * (1.0 if x2 is None else x2.double())
    assert ((out.double() - ref).abs() <= _bound(y, u, D, x2)).all()


def test_medium_filter_keeps_infinities_where_the_multiply_adds_keep_them():
    from uplifting_biomolecular_modeling_b200.ops import seq
    g = _gen(5)
    L, d, K = 1200, 40, 128
    u = torch.randn(1, L, d, device="cuda", generator=g).bfloat16()
    u[0, 300, 3], u[0, 700, 9], u[0, 1199, 0] = float("inf"), float("nan"), float("-inf")
    x2 = torch.ones_like(u)
    h = torch.randn(d, K, device="cuda", generator=g).bfloat16()
    D = torch.zeros(d, device="cuda")
    ht = seq.taps_major(h)
    a = seq.fir_inner_gate(u, ht, D, x2, taps_bf16=True)
    b = seq.fir_inner_gate(u, ht, D, x2)
    assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
    ok = b.isfinite()
    assert (a[ok].double() - b[ok].double()).abs().max() <= 2.0 ** -7 * b[ok].double().abs().max()


@pytest.mark.parametrize("kind", ["hcm", "hcl"])
def test_operator_prefill_matches_its_plain_statement(kind):
    from uplifting_biomolecular_modeling_b200.models import evo2
    torch.manual_seed(3)
    cfg = evo2.CONFIGS["evo2_7b"].__class__(d_model=128, n_heads=1, ffn=256)
    op = evo2.HyenaOperator(cfg, kind).cuda().bfloat16().eval().requires_grad_(False)
    x = torch.randn(2, 700, 128, device="cuda").bfloat16()
    want_s, got_s = {}, {}
    want = op(x, want_s, evo2.fused_linear)
    op.impl = "fused"
    got = op(x, got_s, evo2.fused_linear)
    # bf16 roundings before the output projection and in the plain statement's intermediates
    assert (got.float() - want.float()).norm() <= 2e-2 * want.float().norm()
    assert set(got_s) == set(want_s)
    for k in got_s:
        assert got_s[k].shape == want_s[k].shape and got_s[k].dtype == want_s[k].dtype
        assert (got_s[k].float() - want_s[k].float()).norm() <= 2e-2 * want_s[k].float().norm()
