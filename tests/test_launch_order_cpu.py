"""Where kernels that hold tensor memory let the next kernel of the stream in, read from their sources.

A kernel that is let in early and shares an SM takes its columns and waits for the one in front to end.  So the one in front has to have
its own columns first, in every CTA: its trigger stands behind the barrier that publishes their address."""
import pathlib
import re

import pytest

import uplifting_biomolecular_modeling_b200 as package

SOURCES = sorted((pathlib.Path(package.__file__).parent / "ops" / "csrc").glob("*.cu"))
TRIGGER = re.compile(r"grid_dependency_sync\(|grid_dependency_next\(|griddepcontrol\.launch_dependents")


def _functions(text):
    text = re.sub(r"//[^\n]*", "", text)
    starts = [m.start() for m in re.finditer(r"^(?:__global__|__device__|static |inline |extern |template )", text, re.M)]
    return [text[a:b] for a, b in zip(starts, starts[1:] + [len(text)])]


def _holding(path):
    return [f for f in _functions(path.read_text()) if re.search(r"\btmem_alloc(_pair)?\(", f)]


def test_the_kernels_are_found():
    found = {p.stem: len(_holding(p)) for p in SOURCES}
    assert {k for k, n in found.items() if n} >= {"atom_proj_sm100", "attention_sm100", "gemm_sm100", "pair_proj_sm100", "pwa_sm100",
                                                  "transition_sm100", "trimul_out_sm100", "trimul_proj_sm100"}
    assert found["atom_proj_sm100"] == found["pwa_sm100"] == 2


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.stem)
def test_the_next_kernel_comes_in_behind_the_columns(path):
    for f in _holding(path):
        published = f.index("__syncthreads()", max(m.end() for m in re.finditer(r"\btmem_alloc(_pair)?\(", f)))
        assert all(m.start() > published for m in TRIGGER.finditer(f)), f[:200]
