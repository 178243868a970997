"""What the kernels' sources must say about programmatic dependent launch: a wrong order of trigger, wait and loads is a race that a
run on a GPU hardly ever shows."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "strict_b200", "csrc")


def kernels():
    """{name: (file, parameter list, body)} of every __global__ function, comments taken out."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\(([^{;]*)\)\s*\{", text):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            out[m.group(1)] = (os.path.basename(path), m.group(2), text[m.end():end])
    return out


KERNELS = kernels()


def test_kernels_are_found():
    assert len(KERNELS) > 60 and "quantize_rows_kernel" in KERNELS and "gemm_f32_tc_kernel" in KERNELS


@pytest.mark.parametrize("name", ["quantize_rows_kernel", "quantize_rows_int8_kernel", "quantize_rows_int8_wide_kernel"])
def test_row_splits_trigger_after_their_wait(name):
    """The product behind a split reads weights before its own wait: it may start only when what came before the split, which may
    have written them, is complete."""
    body = KERNELS[name][2]
    assert 0 <= body.index("pdl_wait()") < body.index("pdl_trigger()")
