"""Kernels that start while the one before still runs (programmatic dependent
launch) read nothing of earlier kernels before they have waited for them.  The
compiler may load through a `const T *__restrict__` parameter of a kernel ahead of
the wait, so such a kernel takes none but what is laid out with the mesh; its inputs
are plain pointers (or reach a function with __restrict__ parameters after the
wait)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rheotool_gb300", "csrc")
WITH_THE_MESH = {"cellAt"}


def kernels():
    """(file, name, parameters, body) of every __global__ function."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*\([^{;]*?\)\s+)?(\w+)\s*\(", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            params, j = text[m.end():i - 1], text.index("{", i)
            depth, k = 1, j + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[k], 0)
                k += 1
            yield os.path.basename(path), m.group(1), params, text[j:k]


def dependent():
    return [(f, n, p) for f, n, p, b in kernels() if "after_previous(" in b or "wait_for_previous(" in b]


def test_the_kernels_are_found():
    names = {n for _, n, _ in dependent()}
    assert {"k_tile_sweep", "k_level_apply", "k_level_factor", "k_mg_smooth", "k_pcg_step", "k_bicg_update"} <= names


@pytest.mark.parametrize("file,name,params", dependent(), ids=lambda v: v if str(v).startswith("k_") else "")
def test_no_restrict_inputs(file, name, params):
    inputs = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params))
    assert inputs <= WITH_THE_MESH, (file, name, inputs)
