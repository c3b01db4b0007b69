"""Kernels launched programmatically start while the kernel that writes their inputs still runs.

A `__restrict__` pointer parameter tells the compiler that nothing else touches the object while
the kernel runs: it may load from it before the wait, through the read-only path.  So no kernel
that waits inside takes one."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "crysscft_sample_b200", "csrc")


def _matching(text, i, opening, closing):
    """The index past the bracket that closes the one at i."""
    depth = 0
    for j in range(i, len(text)):
        depth += (text[j] == opening) - (text[j] == closing)
        if depth == 0:
            return j + 1
    raise ValueError("unbalanced")


def _kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s*", text):
            i = m.end()
            if text.startswith("__launch_bounds__", i):
                i = _matching(text, text.index("(", i), "(", ")")
            i = text.index("(", i)
            name = text[m.end():i].split()[-1]
            end = _matching(text, i, "(", ")")
            body = text[text.index("{", end):]
            yield os.path.basename(path), name, text[i:end], body[:_matching(body, 0, "{", "}")]


WAITING = [k for k in _kernels() if "pdl_wait()" in k[3]]


def test_the_waiting_kernels_are_found():
    assert {"prep_kernel", "energy_kernel", "anderson_update_kernel", "axis_mma_kernel", "contour_any_kernel",
            "contour_step_kernel_f32", "contour_simt_kernel_f32"} <= {k[1] for k in WAITING}


@pytest.mark.parametrize("file,name,params,body", WAITING, ids=[k[1] for k in WAITING])
def test_a_waiting_kernel_promises_nothing_about_its_inputs(file, name, params, body):
    assert "__restrict__" not in params
