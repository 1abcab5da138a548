"""Which tiles a GEMM call takes, asked of the library without a launch (and without a GPU: it then counts 148 SMs)."""
import pytest
import torch

from uplifting_biomolecular_modeling_b200.ops import gemm as G
from uplifting_biomolecular_modeling_b200.ops import native

NARROW, WIDE, PAIR, TRIPLE, BOXES = 0, 1, 2, 3, 8


@pytest.fixture
def tiles(monkeypatch):
    if not native.library_path().exists():
        pytest.skip("kernel library not built")
    real = native.lib()
    seen = []

    class Asked:
        @staticmethod
        def ubm_gemm_bf16_packed(args):
            seen.append(real.ubm_gemm_bf16_tiles(args))
            return 0

    monkeypatch.setattr(native, "lib", lambda: Asked)
    monkeypatch.setattr(native, "status_tensor", lambda device: torch.zeros(4, dtype=torch.int32))
    monkeypatch.setattr(native, "current_stream", lambda device=None: 0)

    def ask(a, b, **kw):
        G.gemm(a, b, **kw)
        return seen.pop()
    return ask


def _bf(*shape):
    return torch.empty(shape, dtype=torch.bfloat16)


@pytest.mark.parametrize("K", [648, 704, 768, 896, 904, 1024, 1032, 2048, 2056])
@pytest.mark.parametrize("form,longest", [("plain", 640), ("fp32", 640), ("swiglu", 640), ("bias", 896), ("residual", 896),
                                          ("silu", 896), ("part", 896), ("gate", 1024), ("gelu", 2048)])
def test_pairs_are_left_where_the_epilogue_bounds(tiles, form, longest, K):
    M, N = 7680, 4096                                          # seven waves of 128 x 256 tiles
    a, b = _bf(M, K), _bf(N, K)
    kw = {"plain": {}, "fp32": {"out_dtype": torch.float32}, "swiglu": {"act": "swiglu"}, "bias": {"bias": torch.zeros(N)},
          "residual": {"residual": _bf(M, N)}, "silu": {"act": "silu"}, "gelu": {"act": "gelu"},
          "part": {"act": "sigmoid", "act_from": 3072, "bias": torch.zeros(N)},
          "gate": {"gate": _bf(M, N), "residual": _bf(M, N)}}[form]
    assert tiles(a, b, **kw) == (PAIR if K > longest else WIDE)


@pytest.mark.parametrize("n,ld,want", [(672, 672, PAIR), (688, 688, PAIR), (696, 704, WIDE), (704, 704, WIDE), (712, 720, PAIR),
                                       (768, 768, PAIR), (640, 640, WIDE)])
def test_boxes_of_the_blocked_output(tiles, n, ld, want):
    """The contraction of pair-weighted averaging: 128 sequences are enough tiles for boxes, planes with rows of ld elements."""
    S = 128
    w, v = _bf(8, n, ld)[:, :, :n], _bf(8, S * 32, ld)[:, :, :n]
    out = _bf(n * S * 256)
    assert tiles(w, v, out=out, c_blocked=(32 * S * 256, S * 256, 256), c_batch=32) == want + BOXES


@pytest.mark.parametrize("M,N,K,want", [(7680, 3072, 768, WIDE), (3000, 5760, 1920, PAIR), (3000, 5760, 1528, WIDE),
                                        (129, 12288, 4096, PAIR), (256, 9600, 3072, PAIR), (256, 9600, 3064, WIDE),
                                        (257, 9600, 3072, WIDE), (400, 12288, 4096, PAIR), (200, 12288, 4096, PAIR),
                                        (8192, 128, 4096, NARROW), (1300, 4096, 2040, NARROW), (1300, 4096, 2048, PAIR)])
def test_waves(tiles, M, N, K, want):
    assert tiles(_bf(M, K), _bf(N, K)) == want


def test_other_forms(tiles):
    assert tiles(_bf(64, 128), _bf(192, 128), act="swiglu3") == TRIPLE
    assert tiles(_bf(64, 128), _bf(64, 128), act="swiglu") == WIDE
    assert tiles(_bf(64, 8), _bf(64, 136), mn_major=True) == NARROW
