"""LayerNorm of wide rows: edges of its 256-channel chunks, scales on every alignment, rows that leave a block part empty."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1, 4])
@pytest.mark.parametrize("R,C", [(1, 264), (9, 512), (133, 520), (64, 1024), (17, 1032), (33, 1280), (8, 1288), (15, 2048)])
def test_wide_rows(R, C, offset):
    from uplifting_biomolecular_modeling_b200.ops import rows
    g = torch.Generator(device="cuda").manual_seed(R + C)
    x = (torch.randn(R, C, device="cuda", generator=g) + 0.5).bfloat16()
    flat = torch.randn(2, C + offset, device="cuda", generator=g)
    gamma, beta = torch.empty(C + offset, device="cuda"), torch.empty(C + offset, device="cuda")
    gamma, beta = gamma[offset:].copy_(1 + 0.1 * flat[0, offset:]), beta[offset:].copy_(0.1 * flat[1, offset:])
    xd = x.double()
    unit = (xd - xd.mean(-1, keepdim=True)) * (xd.var(-1, unbiased=False, keepdim=True) + 1e-5).rsqrt()
    for w, b in [(gamma, beta), (gamma, None), (None, None)]:
        want = unit * (1 if w is None else w.double()) + (0 if b is None else b.double())
        got = rows.layernorm_rows(x, w, b).double()
        # one rounding to bf16; the statistics are fp32 sums of at most 2048 values
        assert ((got - want).abs() <= 2 ** -8 * want.abs() + 1e-5).all()
