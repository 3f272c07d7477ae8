"""The kernels start while the one before them in the stream still runs
(csrc/launch.h), and read-only loads are for data that nobody writes during a
kernel's life.  So in every kernel a `const T* __restrict__` parameter is one of the
arrays that are final before the kernel before it started: the plan and the pattern,
A's values and, in a solve, the factor and the right-hand sides; and __ldg reads only
those.  (Checked on the sources: a violation shows as a stale value once in many runs,
or never on the compiler at hand.)
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "taucs_b200", "csrc")
PLAN = {"list", "fronts", "children", "child_rec", "maps", "rows", "acol_ptr", "a_rows", "a_idx", "cum", "tasks",
        "parent_task", "tiles", "tile_ch", "blocks", "pending0", "diagpos", "rowind", "colidx", "rp", "ci", "vi", "seg",
        "vmap", "perm", "vals"}
FINAL = {"numeric.cu": PLAN, "gemm_tc.cu": PLAN, "refine.cu": PLAN, "solve.cu": PLAN | {"L", "B"}}
# first names of what __ldg reads: plan arrays, and pointers into them
LDG = PLAN | {"mp", "rw", "rec"}


def kernels(text):
    for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i - 1]


@pytest.mark.parametrize("name", sorted(FINAL))
def test_read_only_pointers_are_final(name):
    text = open(os.path.join(CSRC, name)).read()
    found = dict(kernels(text))
    assert found
    for kernel, params in found.items():
        for q in re.findall(r"const\s+\w+\*\s*__restrict__\s+(\w+)", params):
            assert q in FINAL[name], (kernel, q)
    for q in re.findall(r"__ldg\(\s*(?:__ldg\(\s*)?(?:A\.)?(\w+)", text):
        assert q in LDG, q


def test_the_check_finds_one():
    bad = "template <typename T>\n__global__ void __launch_bounds__(128)\nk_x(int n, const T* __restrict__ W, (int) 1) {"
    (name, params), = kernels(bad)
    assert name == "k_x" and re.findall(r"const\s+\w+\*\s*__restrict__\s+(\w+)", params) == ["W"]
