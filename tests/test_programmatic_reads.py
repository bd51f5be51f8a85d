"""The kernels of a recorded iteration are launched programmatically: one is resident while the one before it still writes the
solve's vectors. CUDA's read-only path (__ldg, and what the compiler makes of const __restrict__) asks for data that
nothing writes while the kernel is resident, so those kernels may read only the model's own data through it. The
sources are checked: kernels that take a Ctl, and the device functions they share."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "parts-sim_b200", "csrc")
# the single solve's kernels (the block solve's are launched normally; its shared gather is applyNbr)
FILES = ["solver.cu", "kernels.cuh", "march_kernels.cuh", "stencil_kernels.cuh", "ebe_kernels.cuh"]
# parameters and pointers that hold the model's data: masks, words, 1/diag, lists, tiles, matrices, stencils
MODEL = {"nmask", "invD", "list", "tiles", "stn", "dof", "Ainv"}
MODEL_READS = {"L.nmask", "L.word", "L.invD", "C.nmask", "C.invD", "F.nmask", "nmask", "list", "dof", "K4", "K16", "src", "m", "Ainv"}


def text(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def kernels(src):
    """(name, parameter text) of every kernel"""
    for m in re.finditer(r"__global__[^;{]*?(\w+)\((LevelView|int|long long|const)", src):
        end = src.index("{", m.end())
        yield m.group(1), src[m.start(2):end]


@pytest.mark.parametrize("name", FILES)
def test_vectors_of_an_iteration_are_not_declared_read_only(name):
    seen = 0
    for kernel, params in kernels(text(name)):
        if "Ctl ctl" not in params:
            continue
        seen += 1
        for ptr in re.findall(r"const \w+\* __restrict__ (\w+)", params):
            assert ptr in MODEL, (kernel, ptr)
    assert seen > 0 or name == "kernels.cuh"


@pytest.mark.parametrize("name", FILES)
def test_read_only_loads_are_of_the_models_data(name):
    for what in re.findall(r"(?:__ldg|ldModel)\(\s*([A-Za-z_][\w.]*)", text(name)):
        assert what in MODEL_READS or what in MODEL or what == "const", (name, what)  # (const: ldModel's own declarations)


def test_shared_device_functions_take_plain_pointers():
    for name, fn in (("kernels.cuh", "applyAt"), ("block_kernels.cuh", "applyNbr"), ("solver.cu", "restrictAt"), ("solver.cu", "prolongAt")):
        src = text(name)
        at = src.index(f" {fn}(const") if f" {fn}(const" in src else src.index(f" {fn}(long long")
        assert "__restrict__" not in src[at:src.index("{", at)], fn
