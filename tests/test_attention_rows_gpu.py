"""Two-row forms of the attention kernel: groups that are not full (row counts 1 to 7), alone and in front of full ones of the same CTA,
and head dimension 64 without bias in steps of 128 keys, at key counts around its steps."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
LOG2E = 1.4426950408889634


def _case(rows, Nq, Nk, H, D, bias, masked, gated, seed):
    from uplifting_biomolecular_modeling_b200.ops import native, pair
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(s, device="cuda", generator=g)  # noqa: E731
    HD = H * D
    qkvg = r(rows * max(Nq, Nk), 4 * HD).to(BF)
    if Nq == Nk:                                            # column slices of one buffer
        q, k, v, gate = (qkvg[:, i * HD:(i + 1) * HD] for i in range(4))
        ld = 4 * HD
    else:
        q, k, v, gate = (r(rows * n, HD).to(BF) for n in (Nq, Nk, Nk, Nq))
        ld = 0
    gate = torch.sigmoid(gate.float()).to(BF).contiguous() if gated else None
    q = (q.float() * (LOG2E / D ** 0.5)).to(BF).contiguous() if ld == 0 else q
    if ld:
        qkvg[:, :HD] = (qkvg[:, :HD].float() * (LOG2E / D ** 0.5)).to(BF)
    ldb = (Nk + 7) // 8 * 8
    planes = r(H, Nq, ldb).to(BF) if bias else None
    keep = (torch.rand((rows, Nk), device="cuda", generator=g) < 0.7).to(BF) if masked else None
    if masked:
        keep[:, 0] = 1
    out = torch.full((rows * Nq, HD), float("nan"), device="cuda", dtype=BF)
    pair.attention(q, k, v, planes, gate, out, rows=rows, Nq=Nq, Nk=Nk, H=H, D=D, ldb=ldb if bias else 0, ld_in=ld,
                   mask=None if keep is None else pair.KeyMask.lay_out(keep))
    torch.cuda.synchronize()
    native.raise_on_status("cuda", "attention")
    hd = lambda t, n: t.reshape(rows, n, H, D).transpose(1, 2).double()  # noqa: E731
    s = hd(q, Nq) @ hd(k, Nk).transpose(-1, -2)
    if bias:
        s = s + planes[None, :, :, :Nk].double()
    if masked:
        s = s.masked_fill(keep[:, None, None, :] == 0, float("-inf"))
    ref = (torch.softmax(s / LOG2E, -1) @ hd(v, Nk)).transpose(1, 2).reshape(rows * Nq, HD)
    if gated:
        ref = ref * gate.double()
    return ((out.double() - ref).norm() / ref.norm()).item()


# bf16 probabilities (2^-9 each, averaged over the keys) and a bf16 result (2^-9): 4e-3 at most for a handful of keys
@pytest.mark.parametrize("rows", [1, 2, 3, 5, 7])
@pytest.mark.parametrize("D,H,N", [(64, 16, 130), (64, 3, 700), (64, 40, 64), (32, 16, 190)])
def test_groups_that_are_not_full(rows, D, H, N):
    if D == 32 and rows >= 4:
        pytest.skip("head dimension 32 takes groups of four from four rows on")
    assert _case(rows, N, N, H, D, True, False, True, rows + N) < 5e-3
    assert _case(rows, N, N, H, D, True, True, False, rows + N + 1) < 5e-3
    assert _case(rows, N, N, H, D, False, True, False, rows + N + 2) < 5e-3


@pytest.mark.parametrize("rows", [1, 2, 5])
@pytest.mark.parametrize("Nq,Nk", [(1, 1), (5, 5), (127, 127), (128, 128), (129, 129), (300, 64), (64, 257), (513, 513)])
def test_no_bias_in_steps_of_128_keys(rows, Nq, Nk):
    assert _case(rows, Nq, Nk, 15, 64, False, False, Nq == Nk, Nq + Nk) < 5e-3


def _full_after_partial(rows, N, H):
    """Whether some CTA (items blockIdx, + grid, ..) takes a full group of two rows behind one with a missing row."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n_qt, n_rp = -(-N // 128), -(-rows // 2)
    items = n_qt * n_rp * H
    full = lambda item: item // n_qt % n_rp * 2 + 2 <= rows  # noqa: E731
    return any(not full(a) and any(full(b) for b in range(a + sms, items, sms)) for a in range(items))


# an odd number of key steps (five of 64, three of 128), so that a step counted wrongly is a phase counted wrongly
@pytest.mark.parametrize("rows,D,H,bias,masked", [(5, 64, 40, True, False), (5, 64, 40, True, True), (5, 64, 40, False, True),
                                                  (5, 64, 40, False, False), (3, 64, 40, True, True), (3, 32, 40, True, False),
                                                  (3, 32, 40, True, True), (3, 32, 40, False, True)])
def test_full_groups_behind_a_missing_row(rows, D, H, bias, masked):
    N = 300
    assert _full_after_partial(rows, N, H)
    assert _case(rows, N, N, H, D, bias, masked, True, rows + H) < 5e-3


def test_full_groups_behind_a_missing_row_in_steps_of_128_keys():
    from uplifting_biomolecular_modeling_b200.ops import pair
    pair.set_attention_variant(5)
    try:
        assert _full_after_partial(5, 300, 40)
        assert _case(5, 300, 300, 40, 32, True, False, True, 2) < 5e-3
    finally:
        pair.set_attention_variant(0)
