"""Rows that a block of the outer product takes, by its size and by what bounds its memory."""
import pytest
import torch

from uplifting_biomolecular_modeling_b200.models import msa


def _rows(op, N):
    rows, scratch = op._block(N, "meta")
    assert scratch.shape == (rows * N, 1024)
    return rows


@pytest.mark.parametrize("N,rows", [(1, 1), (128, 128), (137, 137), (768, 768), (1024, 1024), (1025, 520), (1100, 552), (4096, 256),
                                    (5000, 200), (8192, 128), (9000, 128)])
def test_as_many_rows_as_the_scratch_holds(N, rows):
    op = msa.OuterProductMean()
    assert _rows(op, N) == rows and rows * N * 2048 <= max(op.SCRATCH, 128 * N * 2048)


@pytest.mark.parametrize("asked", [8, 40, 128, 300])
def test_rows_that_were_asked_for_stay(asked):
    op = msa.OuterProductMean()
    op.row_block = asked
    for N in (20, 137, 768, 4096):
        assert _rows(op, N) == min(asked, N)


def test_row_blocks_of_the_workspace_bound_the_scratch():
    op = msa.OuterProductMean()
    op.set_impl("fused", {"row_block": 512})
    assert _rows(op, 768) == 128 and _rows(op, 100) == 100
    op.set_impl("fused", {"row_block": 0})
    assert _rows(op, 768) == 768
    op.set_impl("fused", {})
    assert _rows(op, 768) == 768


def test_a_shortage_is_met_once(monkeypatch):
    """An allocation that fails empties the allocator's cache; blocks of that size are not asked for again, smaller ones are."""
    op, asked, empty = msa.OuterProductMean(), [], torch.empty

    def short(size, **kw):
        asked.append(size[0])
        if size[0] > 200000:
            raise torch.OutOfMemoryError("no room")
        return empty(size, **kw)

    monkeypatch.setattr(msa.torch, "empty", short)
    assert op._block(600, "meta")[0] == 128 and asked == [600 * 600, 128 * 600]
    asked.clear()
    assert [op._block(N, "meta")[0] for N in (600, 900, 300)] == [128, 128, 300]
    assert asked == [128 * 600, 128 * 900, 300 * 300]
