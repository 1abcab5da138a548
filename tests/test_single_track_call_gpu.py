"""The single track of a Pairformer layer from one call of the library: the same bits, ledger and launch counts as operator by operator,
and operator by operator wherever a call of one of them would do anything else."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _rand(g, *shape):
    return torch.randn(shape, device="cuda", generator=g).to(BF)


def _layer(c=384, heads=16, seed=0):
    from uplifting_biomolecular_modeling_b200.models import pairformer
    torch.manual_seed(seed)
    m = pairformer.PairformerLayer(c, 128, heads).cuda().to(BF).eval().requires_grad_(False)
    for p in m.parameters():
        p.add_(torch.randn_like(p) * 0.02)
    pairformer.set_impl(m, "fused")
    return m


def _apart(m, s, z, mask, monkeypatch):
    from uplifting_biomolecular_modeling_b200.models import pairformer
    with monkeypatch.context() as mp:
        mp.setattr(pairformer.PairformerLayer, "_single_track", lambda self, s, z, mask: None)
        mp.setattr(pairformer.PairformerLayer, "pair_update", lambda self, z, mask: z)
        return m(s, z, mask, None)[0]


@pytest.mark.parametrize("c,heads", [(384, 16), (384, 8), (256, 4), (1024, 16)])
@pytest.mark.parametrize("N,masked", [(1, None), (7, torch.bool), (64, torch.float32), (137, BF), (200, torch.uint8), (201, None)])
def test_single_track_in_one_call(N, masked, c, heads, monkeypatch):
    """Rows that leave a remainder in the sums' eight-element loads, the attention's tiles and the planes' padding; the largest norm."""
    from uplifting_biomolecular_modeling_b200.core import counters
    from uplifting_biomolecular_modeling_b200.ops import native
    m = _layer(c, heads)
    g = torch.Generator(device="cuda").manual_seed(N)
    s, z = _rand(g, 1, N, c) * 30, _rand(g, 1, N, N, 128)
    mask = None
    if masked is not None:
        mask = (torch.rand((1, 2 * N), device="cuda", generator=g) < 0.7).to(masked)[:, ::2]
        mask[:, 0] = 1
    assert m._single_track(s, z, mask) is None                     # not packed yet
    kept = s.clone()
    served = lambda: {k: counters.BOOK.find(k).served for k in ("fused_apb", "fused_transition")}  # noqa: E731
    ref, calls = _apart(m, s, z, mask, monkeypatch), []
    for one in (False, True):
        before = served()
        native.reset_launch_count()
        out = m._single_track(s, z, mask) if one else _apart(m, s, z, mask, monkeypatch)
        calls.append((native.launch_counts(), {k: v - before[k] for k, v in served().items()}))
        assert torch.equal(out, ref) and torch.equal(s, kept)
    own = {k: v for k, v in calls[1][0].items() if k not in ("ubm_single_add", "ubm_single_out")}
    assert (own, calls[1][1]) == calls[0]


def test_values_out_of_range():
    """Infinities and NaN in a row stay in that row's residual and reach what they reached before."""
    m = _layer()
    g = torch.Generator(device="cuda").manual_seed(3)
    s, z = _rand(g, 1, 40, 384), _rand(g, 1, 40, 40, 128)
    for value in (float("inf"), float("nan"), 3e38):
        x = s.clone()
        x[0, 5, 17] = value
        with pytest.MonkeyPatch.context() as mp:
            ref = _apart(m, x, z, None, mp)
        out = m._single_track(x, z, None)
        assert torch.equal(out.isnan(), ref.isnan()) and torch.equal(out.nan_to_num(), ref.nan_to_num())


def test_what_keeps_the_single_track_apart(monkeypatch):
    from uplifting_biomolecular_modeling_b200.models import pairformer
    m = _layer()
    g = torch.Generator(device="cuda").manual_seed(1)
    N = 33
    s, z, mask = _rand(g, 1, N, 384), _rand(g, 1, N, N, 128), torch.ones((1, N), device="cuda", dtype=BF)
    ref = _apart(m, s, z, mask, monkeypatch)
    assert m._single_track(s, z, mask) is not None
    seen = []
    for child in (m.attention, m.transition_s):
        handle = child.register_forward_hook(lambda mod, args, out: seen.append(1))
        assert m._single_track(s, z, mask) is None
        handle.remove()
    whole = torch.nn.modules.module.register_module_forward_pre_hook(lambda mod, args: None)
    assert m._single_track(s, z, mask) is None
    whole.remove()
    old = m.attention.pair_bias
    m.attention.pair_bias = lambda z: old(z)
    assert m._single_track(s, z, mask) is None
    del m.attention.pair_bias
    wide = torch.zeros((1, N, 400), device="cuda", dtype=BF)
    wide[:, :, :384] = s
    assert m._single_track(wide[:, :, :384], z, mask) is None
    assert torch.equal(_apart(m, wide[:, :, :384], z, mask, monkeypatch), ref)
    for other in (mask.double(), torch.ones((1, N + 1), device="cuda"), mask.cpu()):
        assert m._single_track(s, z, other) is None
    assert m._single_track(s.float(), z, mask) is None and m._single_track(torch.cat([s, s]), z, mask) is None
    assert m._single_track(s, z.transpose(1, 2), mask) is None
    with torch.autocast("cuda", dtype=BF):
        assert m._single_track(s, z, mask) is None
    m.pre_norm_s.requires_grad_(True)
    assert m._single_track(s, z, mask) is None
    with torch.no_grad():
        assert torch.equal(m._single_track(s, z, mask), ref)
    m.pre_norm_s.requires_grad_(False)
    m.transition_s.set_impl("reference")
    assert m._single_track(s, z, mask) is None
    pairformer.set_impl(m, "fused")
    assert m._single_track(s, z, mask) is None
