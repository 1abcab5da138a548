"""q and k rows of the encoder: fewer rows than a block's warps, around the resident grid's rows, heads around the 64 channels up to which
lanes share their angles, rotary widths below the head's."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,Dh,rot", [(8, 8, 8), (128, 16, 16), (960, 64, 64), (960, 64, 32), (1024, 128, 128), (256, 256, 64), (1280, 64, 64),
                                      (2048, 64, 64), (512, 128, 0)])
@pytest.mark.parametrize("T", [1, 3, 1775, 1777, 3600])
def test_rows(T, C, Dh, rot):
    from uplifting_biomolecular_modeling_b200.ops import seq
    g = torch.Generator(device="cuda").manual_seed(T + C)
    qkv = (torch.randn(T, 3 * C, device="cuda", generator=g) * 2).bfloat16()
    pos = torch.randint(0, 2048, (T,), device="cuda", generator=g, dtype=torch.int32)
    qg, kg = (torch.rand(C, device="cuda", generator=g) + 0.5 for _ in range(2))
    before = qkv.clone()
    out = seq.qk_norm_rotary_(qkv, pos, qg, kg, C // Dh, rot)
    assert torch.equal(out[:, 2 * C:], before[:, 2 * C:])
    for i, gamma in enumerate((qg, kg)):
        x = torch.nn.functional.layer_norm(before[:, i * C:(i + 1) * C].double(), (C,), gamma.double(), None, 1e-5).view(T, -1, Dh)
        ref = x.clone()
        if rot:
            # the frequency and the angle are fp32 values, as the embedding is defined: both rounded here as well
            freq = (10000.0 ** (-torch.arange(0, rot, 2, device="cuda", dtype=torch.float64) / rot)).float()
            ang = (pos.float()[:, None] * freq).double()[:, None]
            a, b = x[..., 0:rot:2], x[..., 1:rot:2]
            ref[..., 0:rot:2], ref[..., 1:rot:2] = a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()
        got = out[:, i * C:(i + 1) * C].double().view(T, -1, Dh)
        # one rounding to bf16 (2^-8); a frequency two fp32 roundings off turns an angle of up to 2048 by 2048 * 2^-22
        size = x.abs().amax(-1, keepdim=True)
        assert ((got - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -10 * size + 1e-5).all()
