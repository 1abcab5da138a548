"""Pair-weighted averaging and outer-product mean on the kernel path against float64 statements of the modules."""
import pytest
import torch

from uplifting_biomolecular_modeling_b200.ops import reference as R

pytestmark = pytest.mark.gpu


def _module(build, seed):
    torch.manual_seed(seed)
    m = build().cuda()
    with torch.no_grad():
        for p in m.parameters():
            if p.dim() == 1:
                p.copy_(torch.randn_like(p) * 0.2 + (1.0 if p is getattr(m, "norm_m", m.norm if hasattr(m, "norm") else None).weight else 0.0))
    return m.bfloat16().eval().requires_grad_(False)


def _rel(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("S,N,masked,mask_dtype", [(1, 1, False, torch.bfloat16), (3, 40, True, torch.bfloat16),
                                                   (5, 128, False, torch.float32), (2, 129, True, torch.float32),
                                                   (130, 77, True, torch.bfloat16)])
def test_pair_weighted_averaging(S, N, masked, mask_dtype):
    from uplifting_biomolecular_modeling_b200.models import msa, pairformer
    m = _module(msa.PairWeightedAveraging, N)
    pairformer.set_impl(m, "fused")
    x = torch.randn(1, S, N, 64, device="cuda").bfloat16()
    z = torch.randn(1, N, N, 128, device="cuda").bfloat16()
    mask = torch.ones(1, N, N, device="cuda", dtype=mask_dtype)
    if masked:
        mask[:, :, N - N // 5:] = 0
    got = m(x, z, mask)
    d = lambda p: p.detach().double()  # noqa: E731
    want = R.pair_weighted_averaging(x.double(), z.double(), mask.double(), d(m.norm_m.weight), d(m.norm_m.bias),
                                     d(m.norm_z.weight), d(m.norm_z.bias), d(m.proj_m.weight), d(m.proj_g.weight),
                                     d(m.proj_z.weight), d(m.proj_o.weight), m.heads)
    # bias planes, weights, values, averages, gated rows and result are bf16: six roundings of 2^-9, and as much for the
    # gamma-folded weights
    assert got.shape == x.shape and _rel(got, want) <= 12 * 2.0 ** -9
    # a weight written in place counts in the next call
    with torch.no_grad():
        m.proj_o.weight.zero_()
    assert not m(x, z, mask).any()


@pytest.mark.parametrize("S,N,full", [(1, 4, True), (7, 33, False), (64, 130, True), (40, 300, False)])
def test_outer_product_mean(S, N, full):
    from uplifting_biomolecular_modeling_b200.models import msa, pairformer
    m = _module(msa.OuterProductMean, S)
    pairformer.set_impl(m, "fused")
    m.full_mask = full
    x = torch.randn(1, S, N, 64, device="cuda").bfloat16()
    mask = torch.ones(1, S, N, device="cuda", dtype=torch.bfloat16)
    if not full:
        mask = (torch.rand_like(mask, dtype=torch.float32) < 0.8).bfloat16()
    got = m(x, mask)
    d = lambda p: p.detach().double()  # noqa: E731
    want = R.outer_product_mean(x.double(), mask.double(), d(m.norm.weight), d(m.norm.bias), d(m.proj_a.weight),
                                d(m.proj_b.weight), d(m.proj_o.weight), d(m.proj_o.bias))
    # normalised rows, both projections, the product, its projection and the rescaled result are bf16
    assert _rel(got, want) <= 8 * 2.0 ** -9


@pytest.mark.parametrize("M,N,batch", [(1, 32, 1), (33, 96, 3), (200, 320, 8)])
def test_blocked_output_of_a_batch(M, N, batch):
    """Element (b, m, n) of the product at row m, block n // 32, entry b of the output."""
    from uplifting_biomolecular_modeling_b200.ops import gemm
    a = torch.randn(batch, M, 72, device="cuda").bfloat16()
    b = torch.randn(batch, N, 72, device="cuda").bfloat16()
    nb = N // 32
    out = torch.full((M + 1, nb, batch, 32), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm.gemm(a, b, out=out, c_blocked=(32 * nb * batch * 32, nb * batch * 32, batch * 32), c_batch=32)
    want = torch.matmul(a.float(), b.float().transpose(1, 2)).view(batch, M, nb, 32).permute(1, 2, 0, 3)
    assert (out[:M].float() - want).abs().max() <= 2.0 ** -8 * want.abs().max()
    assert (out[M] == 7).all()
