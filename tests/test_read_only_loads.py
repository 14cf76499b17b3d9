"""The step's kernels are resident while the kernel before them still writes (programmatic dependents,
csrc/sdd_internal.cuh), so a read-only load (__ldg, or a const __restrict__ pointer that the compiler turns into
one) of anything that a kernel writes has no defined value.  Read from the sources: in them only the plan's tables
go through __ldg, and no kernel that waits for its predecessor takes a const __restrict__ pointer."""
import glob
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "spectraldoublediffusiveconvection_gb300", "csrc")
#: the plan's tables by the expressions that read them: fixed-point blocks and their exponents (FxRow::load), Dr's rows
#: (diagnostics, right-hand sides), Dr in FP32, the tensor-core operand, the FP32 Linv blocks
TABLES = {"A + (c0 + c) * LD", "fx_row_exp(blk, LD) + r", "fx_col_exp(blk, LD) + 32 * p + lane", "drn + m",
          "a.Dr32 + e", "src + i", "A + (size_t)c * ldl + r"}


def _sources():
    return {os.path.basename(f): open(f).read() for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))}


def _argument(text, start):
    depth, k = 1, start
    while depth:
        depth += {"(": 1, ")": -1}.get(text[k], 0)
        k += 1
    return text[start:k - 1]


def _code(src):
    return re.sub(r"//[^\n]*", "", src)


def test_only_tables_are_read_through_the_read_only_path():
    found = set()
    for name, src in _sources().items():
        code = _code(src)
        for m in re.finditer(r"__ldg\(", code):
            arg = _argument(code, m.end())
            assert arg in TABLES, (name, arg)
            found.add(arg)
        assert "ld.global.nc" not in code, name
    assert found == TABLES


def test_dependent_kernels_take_no_restrict_pointers():
    seen = 0
    for name, src in _sources().items():
        for head, body in re.findall(r"__global__([^{;]*)\{(.*?)\n\}", _code(src), flags=re.S):
            if "after_previous_kernel" in body:
                seen += 1
                assert "__restrict__" not in head, (name, head.strip()[:80])
    assert seen >= 10
