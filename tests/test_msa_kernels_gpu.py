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


def _averaging(seed):
    from uplifting_biomolecular_modeling_b200.models import msa, pairformer
    m = _module(msa.PairWeightedAveraging, seed)
    pairformer.set_impl(m, "fused")
    return m


def _averaging_exact(m, x, z, mask):
    d = lambda p: p.detach().double()  # noqa: E731
    return R.pair_weighted_averaging(x.double(), z.double(), mask.double(), d(m.norm_m.weight), d(m.norm_m.bias),
                                     d(m.norm_z.weight), d(m.norm_z.bias), d(m.proj_m.weight), d(m.proj_g.weight),
                                     d(m.proj_z.weight), d(m.proj_o.weight), m.heads)


@pytest.mark.parametrize("logit", [-3.0, -9.0, -20.0])
def test_pair_weighted_averaging_keeps_small_gates(logit):
    """Gate logits around ``logit``: the gate's error is relative, so the bound is that of any other logits."""
    m = _averaging(3)
    m.norm_m.weight.fill_(1.0)                # folded weights are the weights themselves
    m.norm_m.bias.fill_(0.5)
    m.proj_g.weight.copy_(torch.randn_like(m.proj_g.weight) * 2.0 ** -6 + logit / 32)
    x = torch.randn(1, 4, 50, 64, device="cuda").bfloat16()
    z = torch.randn(1, 50, 50, 128, device="cuda").bfloat16()
    mask = torch.ones(1, 50, 50, device="cuda")
    assert _rel(m(x, z, mask), _averaging_exact(m, x, z, mask)) <= 12 * 2.0 ** -9


def test_pair_weighted_averaging_of_rows_with_a_large_mean():
    """Rows 1004 but for one channel of 1008: the mean is 2000 standard deviations.  Besides the bf16 roundings, fp32
    sums of 64 products of 1004 and a weight below 1/2, divided by the deviation of 1/2: 64 * 2^-24 * 2000 < 2^-7."""
    m = _averaging(4)
    x = torch.full((1, 5, 60, 64), 1004.0, device="cuda")
    x.scatter_(-1, torch.randint(0, 64, (1, 5, 60, 1), device="cuda"), 1008.0)
    x = x.bfloat16()
    z = torch.randn(1, 60, 60, 128, device="cuda").bfloat16()
    mask = torch.ones(1, 60, 60, device="cuda")
    assert _rel(m(x, z, mask), _averaging_exact(m, x, z, mask)) <= 12 * 2.0 ** -9 + 2.0 ** -7


def test_pair_weighted_averaging_refuses_a_mask_on_the_host():
    m = _averaging(5)
    x, z = torch.randn(1, 2, 20, 64, device="cuda").bfloat16(), torch.randn(1, 20, 20, 128, device="cuda").bfloat16()
    with pytest.raises((ValueError, RuntimeError)):
        m(x, z, torch.ones(1, 20, 20))


def test_pair_weighted_averaging_weights_count_however_written():
    m = _averaging(6)
    x, z = torch.randn(1, 3, 40, 64, device="cuda").bfloat16(), torch.randn(1, 40, 40, 128, device="cuda").bfloat16()
    mask = torch.ones(1, 40, 40, device="cuda")
    m(x, z, mask)
    for p in (m.norm_m.weight, m.norm_m.bias, m.proj_m.weight, m.proj_g.weight, m.proj_o.weight):
        p.data.mul_(0.5)                      # in place, without a new version of the parameter
        assert _rel(m(x, z, mask), _averaging_exact(m, x, z, mask)) <= 12 * 2.0 ** -9


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
@pytest.mark.parametrize("norm", ["weight and bias", "weight", "neither"])
def test_parameters_of_pair_weighted_averaging(dtype, norm):
    """Parameter types other than the module's, weights in other strides, a LayerNorm without a bias or without either."""
    from uplifting_biomolecular_modeling_b200.ops import pair
    g = torch.Generator(device="cuda").manual_seed(7)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    S, N = 5, 72
    wm, wg, wo = (r(64, 256) / 8).to(dtype).t(), (r(256, 64) / 8).to(dtype), (r(64, 256) / 16).to(dtype)
    nw, nb = (1 + 0.2 * r(64)).to(dtype), (0.2 * r(64)).to(dtype)
    nw, nb = nw if norm != "neither" else None, nb if norm == "weight and bias" else None
    m, planes = r(S, N, 64).bfloat16(), r(8, N, N).bfloat16()
    w = torch.softmax(planes.double(), -1)
    d = lambda t: None if t is None else t.double()  # noqa: E731
    n = torch.nn.functional.layer_norm(m.double(), (64,), d(nw), d(nb), 1e-5)
    o = torch.einsum("hij,sjhc->sihc", w, (n @ d(wm).t()).view(S, N, 8, 32)).reshape(S, N, 256)
    want = (torch.sigmoid(n @ d(wg).t()) * o) @ d(wo).t()
    got = pair.pair_weighted_averaging_fused(m, planes.clone(), None, pair.PwaPacked.pack(nw, nb, wm, wg, wo, 1e-5))
    assert _rel(got, want) <= 12 * 2.0 ** -9


@pytest.mark.parametrize("name", ["proj_m", "proj_g", "proj_o"])
def test_projections_of_pair_weighted_averaging_are_called(name):
    """A hook on a projection, and another module in its place, take part in the call; gradients are recorded."""
    m = _averaging(8)
    x, z = torch.randn(1, 3, 40, 64, device="cuda").bfloat16(), torch.randn(1, 40, 40, 128, device="cuda").bfloat16()
    mask = torch.ones(1, 40, 40, device="cuda")
    lin = getattr(m, name)
    handle = lin.register_forward_hook(lambda mod, args, y: y * 2)
    hooked = m(x, z, mask)
    handle.remove()
    setattr(m, name, torch.nn.Sequential(lin))
    replaced = m(x, z, mask)
    setattr(m, name, lin)
    plain = m(x, z, mask)
    assert _rel(replaced, plain.double()) <= 12 * 2.0 ** -9
    lin.weight.data.mul_(2)                   # what the hook did
    assert _rel(hooked, m(x, z, mask).double()) <= 12 * 2.0 ** -9
    assert _rel(hooked, plain.double()) > 0.1
    if name != "proj_m":                      # its product is an operand of a kernel that records nothing
        lin.weight.requires_grad_(True)
        m(x, z, mask).float().sum().backward()
        assert lin.weight.grad is not None and lin.weight.grad.abs().sum() > 0


@pytest.mark.parametrize("name", ["proj_a", "proj_b"])
def test_projections_of_the_outer_product_mean_are_called(name):
    from uplifting_biomolecular_modeling_b200.models import msa, pairformer
    m = _module(msa.OuterProductMean, 9)
    pairformer.set_impl(m, "fused")
    x = torch.randn(1, 6, 40, 64, device="cuda").bfloat16()
    mask = torch.ones(1, 6, 40, device="cuda")
    lin = getattr(m, name)
    plain = m(x, mask)
    handle = lin.register_forward_hook(lambda mod, args, y: y * 0)
    # nothing is left but the bias, rounded to bf16 in the kernel's output
    assert torch.equal(m(x, mask), m.proj_o.bias.expand_as(plain))
    handle.remove()
    setattr(m, name, torch.nn.Sequential(lin))
    assert _rel(m(x, mask), plain.double()) <= 8 * 2.0 ** -9


def test_outer_product_mean_with_a_mask_that_broadcasts_over_tokens():
    from uplifting_biomolecular_modeling_b200.models import msa, pairformer
    m = _module(msa.OuterProductMean, 10)
    pairformer.set_impl(m, "fused")
    x = torch.randn(1, 6, 40, 64, device="cuda").bfloat16()
    rows = (torch.arange(6, device="cuda") < 4).float().view(1, 6, 1)
    assert torch.equal(m(x, rows), m(x, rows.expand(1, 6, 40).contiguous()))


@pytest.mark.parametrize("S,N", [(700, 129), (1000, 40)])
def test_pair_weighted_averaging_with_many_tiles_per_cta(S, N):
    """1400 and 1000 tiles of 128 tokens: both teams of the output stage, every buffer, ring slot and phase of the two
    persistent kernels come round several times, with a ragged last tile in each sequence."""
    from uplifting_biomolecular_modeling_b200.ops import native
    m = _averaging(S)
    x = torch.randn(1, S, N, 64, device="cuda").bfloat16()
    z = torch.randn(1, N, N, 128, device="cuda").bfloat16()
    mask = torch.ones(1, N, N, device="cuda")
    mask[:, :, N - 3:] = 0
    got, again = m(x, z, mask), m(x, z, mask)
    native.raise_on_status("cuda", "pair-weighted averaging")
    assert torch.equal(got, again)
    want = _averaging_exact(m, x, z, mask)
    assert _rel(got, want) <= 12 * 2.0 ** -9
    # row by row, so that one wrong tile shows: a row's 64 values share the roundings above
    assert ((got.double() - want).norm(dim=-1) <= 0.1 * want.norm(dim=-1) + 0.02 * want.norm(dim=-1).mean()).all()


def test_blocked_output_of_a_batch_with_many_tiles():
    """At least 384 output tiles: several per CTA, so that the staging of the stores is reused."""
    from uplifting_biomolecular_modeling_b200.ops import gemm
    batch, M, N = 8, 3003, 320
    a = torch.randn(batch, M, 72, device="cuda").bfloat16()
    b = torch.randn(batch, N, 72, device="cuda").bfloat16()
    nb = N // 32
    out = torch.full((M + 1, nb, batch, 32), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm.gemm(a, b, out=out, c_blocked=(32 * nb * batch * 32, nb * batch * 32, batch * 32), c_batch=32)
    want = torch.matmul(a.float(), b.float().transpose(1, 2)).view(batch, M, nb, 32).permute(1, 2, 0, 3)
    assert (out[:M].float() - want).abs().max() <= 2.0 ** -8 * want.abs().max()
    assert (out[M] == 7).all()
