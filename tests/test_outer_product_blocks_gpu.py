"""Row blocks of the outer product: whole, several with a shorter last one, a given size, and the small ones where memory is short."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("N", [1, 7, 64, 137, 200, 301])
def test_blocks(N, monkeypatch):
    from uplifting_biomolecular_modeling_b200.models import msa, pairformer
    torch.manual_seed(N)
    op = msa.OuterProductMean().cuda().to(BF).requires_grad_(False)
    pairformer.set_impl(op, "fused")
    m = torch.randn(1, 12, N, 64, device="cuda").to(BF)
    mask = (torch.rand(1, 12, N, device="cuda") < 0.8).to(BF)
    assert op._block(N, "cuda")[0] == N
    ref = op(m, mask)
    for scratch in (0, 150 * N * 2048, 1 << 40):
        monkeypatch.setattr(msa.OuterProductMean, "SCRATCH", scratch)
        rows, t2 = op._block(N, "cuda")
        assert t2.shape == (rows * N, 1024) and rows <= N and rows * N * 2048 <= max(scratch + 8 * N * 2048, 128 * N * 2048)
        assert torch.equal(op(m, mask), ref)
    op.row_block = 40                                      # a size that was asked for stays
    assert op._block(N, "cuda")[0] == min(40, N) and torch.equal(op(m, mask), ref)


def test_short_of_memory(monkeypatch):
    from uplifting_biomolecular_modeling_b200.models import msa, pairformer
    torch.manual_seed(0)
    op = msa.OuterProductMean().cuda().to(BF).requires_grad_(False)
    pairformer.set_impl(op, "fused")
    m, mask = torch.randn(1, 5, 300, 64, device="cuda").to(BF), torch.ones(1, 5, 300, device="cuda", dtype=BF)
    ref, empty = op(m, mask), torch.empty

    def short(*size, **kw):
        if size and size[0] == (300 * 300, 1024):
            raise torch.OutOfMemoryError("no room")
        return empty(*size, **kw)

    monkeypatch.setattr(msa.torch, "empty", short)
    assert op._block(300, "cuda")[0] == 128 and torch.equal(op(m, mask), ref)


@pytest.mark.parametrize("N,scratch,blocks", [(301, 200 * 301 * 2048, [152, 149]), (425, 144 * 425 * 2048, [144, 144, 137]),
                                              (1100, None, [552, 548])])
def test_equal_blocks_with_a_shorter_last_one(N, scratch, blocks, monkeypatch):
    """More than one block, each larger than 128 rows: the last one writes part of the scratch."""
    from uplifting_biomolecular_modeling_b200.models import msa, pairformer
    torch.manual_seed(N)
    op = msa.OuterProductMean().cuda().to(BF).requires_grad_(False)
    pairformer.set_impl(op, "fused")
    m = torch.randn(1, 12, N, 64, device="cuda").to(BF)
    mask = (torch.rand(1, 12, N, device="cuda") < 0.8).to(BF)
    op.row_block = 128
    ref = op(m, mask)
    op.row_block = None
    if scratch is not None:
        monkeypatch.setattr(msa.OuterProductMean, "SCRATCH", scratch)
    rows = op._block(N, "cuda")[0]
    assert [min(rows, N - i) for i in range(0, N, rows)] == blocks
    assert torch.equal(op(m, mask), ref)
