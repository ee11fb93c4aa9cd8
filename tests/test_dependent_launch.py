"""Kernels under programmatic dependent launch begin while their predecessor
runs, so what that one writes may not be read through the read-only path
(__ldg, const __restrict__ parameters): those loads are for memory that does
not change during the kernel's lifetime, and pdl_wait does not order them.
A check of the sources, since the fault would show as a rare wrong value."""
import glob
import os
import re

import pytest

from exadglm_b200 import build as _build

# members of the argument structs (and pointers into them) that kernels write
WRITTEN = re.compile(r"\b(a\.(u_in|u_out|tau|maxv|kreg|sc)|ubase|kt)\b")


def balanced(text, start, pair="()"):
    """The text from the bracket at `start` to its partner."""
    depth = 0
    for i in range(start, len(text)):
        depth += {pair[0]: 1, pair[1]: -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i + 1]
    raise ValueError("unbalanced")


def kernels(text):
    """(name, parameters, body) of every __global__ function with a body."""
    for m in re.finditer(r"__global__", text):
        k = re.compile(r"(\w+)\s*(\()").search(text, m.end())
        while k.group(1) == "__launch_bounds__":
            k = re.compile(r"(\w+)\s*(\()").search(
                text, k.start(2) + len(balanced(text, k.start(2))))
        params = balanced(text, k.start(2))
        at = k.start(2) + len(params)
        if text[at:].lstrip().startswith("{"):
            yield k.group(1), params, balanced(text, text.index("{", at), "{}")


def source(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


def test_parameters_are_not_restrict():
    seen = 0
    for path in glob.glob(os.path.join(_build.CSRC, "*.cu*")):
        for name, params, body in kernels(source(path)):
            if "pdl_wait()" in body:
                seen += 1
                assert "__restrict__" not in params, (os.path.basename(path), name)
    assert seen >= 9


@pytest.mark.parametrize("name", ["dglm_stage_sym.cuh", "dglm_stage_sym_adv.cuh",
                                  "dglm_stage_tc.cuh", "dglm_stage_tcb.cuh", "dglm_batch.cu"])
def test_written_arrays_are_read_by_plain_loads(name):
    text = source(os.path.join(_build.CSRC, name))
    for m in re.finditer(r"__ldg(?=\()", text):
        arg = balanced(text, m.end())
        assert not WRITTEN.search(arg), arg
