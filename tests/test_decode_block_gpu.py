"""A decoding step of a block from one call: the same bits in output and states as launch by launch, for every operator, and what
keeps it apart."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _model(kinds=None):
    from uplifting_biomolecular_modeling_b200.models import evo2
    cfg = evo2.replace(evo2.CONFIGS["evo2_1b"], n_layers=4, attn_layers=(3,))
    torch.manual_seed(0)
    m = evo2.StripedHyena2(cfg).cuda().to(BF).eval().requires_grad_(False)
    for b in m.blocks:                                      # decays below one
        if hasattr(b.mixer, "log_poles"):
            b.mixer.log_poles.copy_(-torch.rand_like(b.mixer.log_poles.float()).to(BF) - 0.01)
    m.set_impl("fused")
    return m


def _states(m, B, L):
    g = torch.Generator(device="cuda").manual_seed(B + L)
    tokens = torch.randint(0, m.cfg.vocab, (B, L), device="cuda", generator=g)
    states = [{} for _ in m.blocks]
    m(tokens, states)
    m.make_static_states(states, L + 40)
    return states


def _copy(states):
    pos = next(s["pos"] for s in states if "pos" in s).clone()
    return [{k: pos if k == "pos" else v.clone() if torch.is_tensor(v) else v for k, v in s.items()} for s in states]


@pytest.mark.parametrize("B,L", [(1, 5), (1, 1500), (2, 200), (5, 130), (8, 64)])
def test_step_in_one_call(B, L, monkeypatch):
    from uplifting_biomolecular_modeling_b200.models import evo2
    from uplifting_biomolecular_modeling_b200.ops import native
    m = _model()
    start = _states(m, B, L)
    g = torch.Generator(device="cuda").manual_seed(7)
    tokens = torch.randint(0, m.cfg.vocab, (3, B, 1), device="cuda", generator=g)
    runs = []
    for one in (False, True):
        with monkeypatch.context() as mp:
            if not one:
                mp.setattr(evo2.Block, "_step_call", lambda self, x, state, folded: None)
            st = _copy(start)
            native.reset_launch_count()
            logits = [m.step(t, st) for t in tokens]
            runs.append((logits, st, native.launch_counts()))
    for a, b in zip(runs[0][0], runs[1][0]):
        assert torch.equal(a, b)
    for a, b in zip(runs[0][1], runs[1][1]):
        assert a.keys() == b.keys() and all(torch.equal(a[k], b[k]) for k in a if torch.is_tensor(a[k]))
    assert runs[0][2] == runs[1][2]
    assert all(blk._step_call(torch.zeros(B, 1, m.cfg.d_model, device="cuda", dtype=BF), s, m.folded) is not None
               for blk, s in zip(m.blocks, _copy(start)))


def test_what_keeps_a_step_apart():
    m = _model()
    st = _states(m, 2, 40)
    x = torch.zeros(2, 1, m.cfg.d_model, device="cuda", dtype=BF)
    ask = lambda i, s, xx=x, f=None: m.blocks[i]._step_call(xx, s, f or m.folded)  # noqa: E731
    other = lambda *a, **k: m.folded(*a, **k)  # noqa: E731
    for i in range(4):
        fresh = lambda: {k: v.clone() if torch.is_tensor(v) else v for k, v in st[i].items()}  # noqa: E731
        assert ask(i, fresh()) is not None
        assert ask(i, fresh(), f=other) is None
        s = fresh()
        s["static"] = False
        assert ask(i, s) is None
        assert ask(i, fresh(), xx=torch.zeros(2, 2, m.cfg.d_model, device="cuda", dtype=BF)[:, ::2]) is None
        name = next(k for k in ("k", "poles", "inner_tail") if k in st[i])
        s = fresh()
        s[name] = s[name].double() if name == "poles" else s[name].float()
        assert ask(i, s) is None
        mix = m.blocks[i].mixer
        mix.step = type(mix).step.__get__(mix)
        assert ask(i, fresh()) is None
        del mix.step
    m.set_fp8_input_projections(True)
    assert ask(0, dict(st[0])) is None
