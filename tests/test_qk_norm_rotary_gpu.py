"""LayerNorm and rotary embedding of q and k in place, against the separate fp32 statements."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,H,Dh,rot", [(1, 2, 32, 32), (9, 15, 64, 64), (130, 18, 64, 48), (33, 24, 64, 64), (8, 1, 64, 0)])
def test_qk_norm_rotary_in_place(T, H, Dh, rot):
    from uplifting_biomolecular_modeling_b200.ops import reference as R, seq
    g = torch.Generator(device="cuda").manual_seed(T)
    C = H * Dh
    qkv = (torch.randn(T, 3 * C, device="cuda", generator=g) * 2 + 0.5).bfloat16()
    qg, kg = (torch.randn(C, device="cuda", generator=g) for _ in range(2))
    pos = torch.randint(0, 5000, (T,), device="cuda", generator=g)
    ln = lambda x, w: torch.nn.functional.layer_norm(x.float(), (C,), w, None, 1e-5)  # noqa: E731
    q, k, v = qkv.split(C, 1)
    want = torch.cat([ln(q, qg), ln(k, kg), v.float()], 1)
    if rot:
        want = torch.cat([t.reshape(T, C) for t in R.rotary_split_qkv(want, pos, H, rot)], 1)
    out = seq.qk_norm_rotary_(qkv, pos, qg, kg, H, rot)
    assert out is qkv
    # one bf16 rounding per value, and the fp32 angle of a position p carries an error of p * 2^-24
    err = (out.float() - want).abs()
    assert (err <= 2.0 ** -8 * want.abs() + 5000 * 2.0 ** -22 * want.abs().max()).all()
