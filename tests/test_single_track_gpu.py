"""The single track of a Pairformer layer when its attention falls back to the plain statements."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def layer(monkeypatch):
    from uplifting_biomolecular_modeling_b200.models import pairformer
    from uplifting_biomolecular_modeling_b200.ops import dispatch, provider
    monkeypatch.setitem(dispatch._GATES, "fused_apb", provider.SizeGate("fused_apb", min_tokens=1000, max_tokens=None))
    torch.manual_seed(0)
    m = pairformer.PairformerLayer().cuda().bfloat16().eval()
    pairformer.set_impl(m, "fused")
    return m


def _inputs(n=40):
    return torch.randn(1, n, 384, device="cuda").bfloat16(), torch.randn(1, n, n, 128, device="cuda").bfloat16()


def test_the_callers_autocast_does_not_reach_it(layer):
    seen = []
    layer.attention.register_forward_hook(lambda *a: seen.append(torch.is_autocast_enabled("cuda")))
    s, z = _inputs()
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.float16):
        layer(s, z, None, None)
    assert seen == [False]


def test_gradients_of_its_norm_are_recorded(layer):
    s, z = _inputs()
    layer.requires_grad_(False)
    layer.pre_norm_s.requires_grad_(True)
    out, _ = layer(s, z, None, None)
    out.float().sum().backward()
    assert layer.pre_norm_s.weight.grad is not None and layer.pre_norm_s.weight.grad.abs().sum() > 0


def test_both_forms_of_the_norm_agree(layer):
    """Without a gradient the normalised rows come from one launch: one rounding to bf16 after fp32 arithmetic, as in the
    other form."""
    s, z = _inputs()
    layer.requires_grad_(False)
    seen = []
    layer.attention.register_forward_hook(lambda mod, args, y: seen.append(args[0]))
    with torch.no_grad():
        layer(s, z, None, None)
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        layer(s, z, None, None)
    a, b = (t.float() for t in seen)
    assert seen[0].dtype == seen[1].dtype == torch.bfloat16
    assert ((a - b).abs() <= 2.0 ** -7 * b.abs() + 2.0 ** -20).all()
