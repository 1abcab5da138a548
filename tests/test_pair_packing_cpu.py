"""Packed weights of the pair kernels, evaluated on the CPU the way the kernels read them."""
import pytest
import torch
import torch.nn.functional as F

from uplifting_biomolecular_modeling_b200.ops import native, pair
from uplifting_biomolecular_modeling_b200.ops import reference as R


@pytest.mark.parametrize("hidden", [64, 128, 192])
def test_transition_weights_in_chunks_of_the_kernel(hidden):
    g = torch.Generator().manual_seed(hidden)
    r = lambda *s: torch.randn(*s, generator=g, dtype=torch.float64)  # noqa: E731
    # weights and gamma that are bf16 values with a bf16 product, so that the packed form is exact
    bf = lambda t: t.bfloat16().double()  # noqa: E731
    nw, nb = torch.full((128,), 0.5, dtype=torch.float64), bf(r(128))
    a, b, o = bf(r(hidden, 128)), bf(r(hidden, 128)), bf(r(128, hidden))
    x = r(9, 128)
    w = pair.TransitionPacked.pack(nw, nb, a, b, o)
    assert w.hidden >= 128 and w.hidden % 64 == 0
    assert w.wab.shape == (2 * w.hidden, 128) and w.wo.shape == (128, w.hidden)
    assert w.colsum.shape == w.colbias.shape == (2 * w.hidden,)
    assert all(t.is_contiguous() for t in (w.wab, w.wo, w.colsum, w.colbias))
    mu, rstd = x.mean(-1, keepdim=True), torch.rsqrt(x.var(-1, unbiased=False, keepdim=True) + 1e-5)
    y = torch.zeros(9, 128, dtype=torch.float64)
    for c in range(w.hidden // 64):
        at = slice(128 * c, 128 * c + 128)
        pre = rstd * (x @ w.wab[at].double().T - mu * w.colsum[at].double()) + w.colbias[at].double()
        y += (F.silu(pre[:, :64]) * pre[:, 64:]) @ w.wo[:, 64 * c:64 * c + 64].double().T
    want = R.transition(x, nw, nb, a, b, o)
    # column sums and biases are fp32
    assert (y - want).abs().max() <= 1e-5 * want.abs().max()


def test_transition_kernel_refuses_a_single_chunk():
    if not native.available():
        pytest.skip("kernel library not built")
    lib = native.lib()
    for hidden in (0, 64, 96, 1088):
        assert lib.ubm_transition(0, 0, 0, 0, 0, 0, 0, 0, 128, hidden, 1, 0, 0) == -1
