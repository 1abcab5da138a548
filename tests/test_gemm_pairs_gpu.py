"""GEMM tiles shared by two SMs: edges of the 256 x 256 tile and of the k-blocks, both operand layouts, batches, every epilogue
and both forms of the blocked output.  The first product of each test is checked to take such tiles (the sizes are for 148 SMs)."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _r(seed, *shape):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, device="cuda", generator=g).bfloat16()


PAIR, BOXES = 2, 8


@pytest.fixture(autouse=True)
def taken(monkeypatch):
    """Tiles of the products of a test."""
    from uplifting_biomolecular_modeling_b200.ops import native
    lib, seen = native.lib(), []

    class Asking:
        def __getattr__(self, name):
            return getattr(lib, name)

        def ubm_gemm_bf16_packed(self, args):
            seen.append(lib.ubm_gemm_bf16_tiles(args))
            return lib.ubm_gemm_bf16_packed(args)

    asking = Asking()
    monkeypatch.setattr(native, "lib", lambda: asking)
    yield seen
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert seen and seen[0] & ~BOXES == PAIR


def _close(got, want):
    # fp32 sums of exact products, one rounding to bf16
    assert (got.double() - want).norm() <= 1.1 * 2.0 ** -9 * want.norm()
    assert not ((got.double() - want).abs() > 2.0 ** -8 * want.abs() + 1e-4 * want.abs().max()).any()


# six waves of a short contraction (the last tile one row, one column high), a few waves of a longer one, 130 to 256 rows
@pytest.mark.parametrize("M,N,K", [(4864, 5128, 648), (12801, 2297, 712), (12673, 2296, 704), (2100, 4616, 2056),
                                   (2049, 4353, 2048), (130, 9608, 3080), (256, 9600, 3072)])
@pytest.mark.parametrize("mn_major", [False, True])
def test_plain(M, N, K, mn_major):
    from uplifting_biomolecular_modeling_b200.ops import gemm, native
    Mp, Np, Kp = (-(-v // 8) * 8 for v in (M, N, K))
    a = _r(M, K, Mp)[:, :M] if mn_major else _r(M, M, Kp)[:, :K]
    b = _r(N, K, Np)[:, :N] if mn_major else _r(N, N, Kp)[:, :K]
    bias, res = torch.randn(N, device="cuda"), _r(5, M, Np)[:, :N]
    prod = (a.double().T @ b.double()) if mn_major else a.double() @ b.double().T
    _close(gemm.gemm(a, b, mn_major=mn_major), prod)
    _close(gemm.gemm(a, b, mn_major=mn_major, bias=bias, residual=res, alpha=0.5), 0.5 * prod + bias.double() + res.double())
    native.raise_on_status("cuda", "gemm")


@pytest.mark.parametrize("n", [641, 897])
@pytest.mark.parametrize("mn_major", [False, True])
def test_batch(n, mn_major):
    from uplifting_biomolecular_modeling_b200.ops import gemm, native
    ld = -(-n // 8) * 8
    a, b = _r(1, 96, n, ld)[:, :, :n], _r(2, 96, n, ld)[:, :, :n]
    out = torch.zeros(96, n, ld, device="cuda", dtype=torch.bfloat16)
    gemm.gemm(a, b, mn_major=mn_major, out=out[:, :, :n])
    native.raise_on_status("cuda", "gemm")
    want = torch.bmm(a.double().transpose(1, 2), b.double()) if mn_major else torch.bmm(a.double(), b.double().transpose(1, 2))
    _close(out[:, :, :n], want)
    assert not out[:, :, n:].any()


@pytest.mark.parametrize("tokens,sequences", [(160, 650)])
def test_blocked_outer_product(tokens, sequences):
    from uplifting_biomolecular_modeling_b200.ops import gemm, native
    a, b = _r(3, sequences, tokens * 32), _r(4, sequences, tokens * 32)
    out = torch.empty(tokens * tokens, 1024, device="cuda", dtype=torch.bfloat16)
    gemm.gemm(a, b, mn_major=True, out=out, c_blocked=(tokens * 1024, 32, 1024))
    native.raise_on_status("cuda", "gemm")
    want = torch.einsum("sic,sjd->ijcd", a.double().view(sequences, tokens, 32), b.double().view(sequences, tokens, 32))
    _close(out, want.reshape(tokens * tokens, 1024))


@pytest.mark.parametrize("M,hidden,K", [(2050, 2048, 1544), (12001, 1056, 648)])
def test_swiglu(M, hidden, K):
    from uplifting_biomolecular_modeling_b200.ops import gemm, native
    x, wg, wv = _r(6, M, K), _r(7, hidden, K) * K ** -0.5, _r(8, hidden, K) * K ** -0.5
    got = gemm.gemm(x, gemm.pack_swiglu(wg, wv), act="swiglu")
    native.raise_on_status("cuda", "gemm")
    want = F.silu(x.double() @ wg.double().T) * (x.double() @ wv.double().T)
    # the gate's sigmoid has a relative error of 2e-4
    assert (got.double() - want).norm() <= 1.5 * 2.0 ** -9 * want.norm()


# one column block of the activation's part, odd numbers of row blocks, one row in the last
@pytest.mark.parametrize("M,N,K", [(4864, 5128, 2056), (2177, 4616, 2120), (130, 9608, 3080)])
@pytest.mark.parametrize("form", ["fp32", "bias_residual", "silu", "sigmoid_from", "gelu", "relu_bias", "gate_residual", "shared_gate"])
def test_epilogues(M, N, K, form):
    from uplifting_biomolecular_modeling_b200.ops import gemm, native
    a, b, bias = _r(11, M, K) * K ** -0.5, _r(12, N, K), torch.randn(N, device="cuda")
    prod, res, gate = a.double() @ b.double().T, _r(14, M, N), _r(15, M, N)
    rows = next(r for r in (65, 7, 19) if M % r == 0) if M % 65 == 0 or M % 7 == 0 or M % 19 == 0 else M
    kw, want = {"fp32": ({"out_dtype": torch.float32}, prod),
                "bias_residual": ({"bias": bias, "residual": res, "alpha": 0.5}, 0.5 * prod + bias.double() + res.double()),
                "silu": ({"act": "silu"}, F.silu(prod)),
                "sigmoid_from": ({"act": "sigmoid", "act_from": 4096}, torch.cat([prod[:, :4096], prod[:, 4096:].sigmoid()], 1)),
                "gelu": ({"act": "gelu"}, F.gelu(prod)),
                "relu_bias": ({"act": "relu", "bias": bias}, F.relu(prod + bias.double())),
                "gate_residual": ({"gate": gate, "residual": res}, prod * gate.double() + res.double()),
                "shared_gate": ({"gate": gate[:rows]}, prod * gate[:rows].double().repeat(M // rows, 1))}[form]
    got = gemm.gemm(a, b, **kw)
    native.raise_on_status("cuda", "gemm")
    assert got.dtype == kw.get("out_dtype", torch.bfloat16)
    # fp32 sums, a rounding to bf16 and, in the activations, tanh.approx (2^-11 of a value to 1, times a value to about 6)
    assert (got.double() - want).norm() <= (1e-5 if form == "fp32" else 1.1 * 2.0 ** -9) * want.norm()
    assert not ((got.double() - want).abs() > 2.0 ** -8 * want.abs() + 6 * 2.0 ** -11).any()


@pytest.mark.parametrize("n,ld", [(649, 656), (712, 720), (897, 904)])
def test_blocked_boxes(taken, n, ld):
    """The contraction of pair-weighted averaging: a batch over heads whose outputs interleave, as bulk copies of 32 x 32 boxes; an
    odd and an even number of 128-row blocks, the last with one row and more."""
    from uplifting_biomolecular_modeling_b200.ops import gemm, native
    S = 133
    w, v = _r(16, 8, n, ld)[:, :, :n], _r(17, 8, S * 32, ld)[:, :, :n]
    out = torch.full((n * S * 256 + 4096,), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm.gemm(w, v, out=out, c_blocked=(32 * S * 256, S * 256, 256), c_batch=32)
    native.raise_on_status("cuda", "gemm")
    assert taken == [PAIR + BOXES]
    got = out[:n * S * 256].view(n, S, 8, 32)
    for h in range(8):
        _close(got[:, :, h].reshape(n, -1), w[h].double() @ v[h].double().T)
    assert (out[n * S * 256:] == 7).all()


@pytest.mark.parametrize("blocks", range(48, 54))
def test_ring_ends_at_any_stage(blocks):
    """One tile per pair that ends at each of the ring's six stages, launched back to back: no commit of a launch may still be
    under way to a CTA that has left."""
    from uplifting_biomolecular_modeling_b200.ops import gemm, native
    M, N, K = 200, 9608, 64 * blocks
    a, b = _r(9, M, K), _r(10, N, K)
    got = [gemm.gemm(a, b) for _ in range(8)]
    native.raise_on_status("cuda", "gemm")
    _close(got[0], a.double() @ b.double().T)
    assert all(torch.equal(g, got[0]) for g in got)
