"""Kernels that may start before the one ahead of them has finished.

Such a kernel (csrc/common.cuh, launch_dependent) must wait before it touches
global memory, and must not promise the compiler that its inputs are constant
for its whole life: the kernel ahead may still be writing them when it starts.
No GPU here: the sources are read.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "daqiri-mixer_b200", "csrc")


def _kernels():
    """{name: (parameters, body)} of every __global__ function."""
    out = {}
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            src = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\(([^{]*)\)\s*\{(.*?)\n\}", src, re.S):
            out[m.group(1)] = (m.group(2), m.group(3))
    return out


def _dependent():
    """Names of the kernels launched by launch_dependent."""
    names = set()
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            src = f.read()
        for m in re.finditer(r"launch_dependent\((?:mixer::)?(\w+)", src):
            k = m.group(1)
            if not k.startswith("k_"):      # a local name for an instance of a template
                found = re.search(r"const auto %s = (k_\w+)<" % k, src)
                if found is None:
                    continue                # the definition of launch_dependent itself
                k = found.group(1)
            names.add(k)
    return sorted(names)


def test_every_dependent_kernel_is_found():
    assert set(_dependent()) == {"k_corner_turn", "k_grid_tiles", "k_image_fft", "k_image_fft_warp",
                                 "k_vis_flush", "k_vis_unpack", "k_xcorr_tri", "k_zero"}


@pytest.mark.parametrize("name", _dependent())
def test_dependent_kernel_waits_and_promises_nothing(name):
    params, body = _kernels()[name]
    assert "pdl_wait()" in body
    assert "__restrict__" not in params
