"""Kernels that start before their predecessor has ended read its results behind a
wait (step_begin).  Their parameters may not be __restrict__ on arrays that a step
writes: the promise would hold from the kernel's start, before the wait, and lets
the compiler read early or through the non-coherent path."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "meshlesshydro_gb300", "csrc")
FIXED = {"members", "memberOf"}     # written when the context is created

KERNEL = re.compile(r"__global__ void [^;{]*?\b(k_\w+)\(([^{]*?)\)\s*\{\s*(\S+)")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def kernels():
    out = {}
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            for m in KERNEL.finditer(source(name)):
                out[m.group(1)] = (m.group(2), m.group(3))
    return out


def launched_early():
    text = source("mlh_kernels.cu")
    names = set(re.findall(r"launch_dep\((k_\w+)", text)) | set(re.findall(r"launch_kernel\(\w+, (k_\w+)", text))
    # kernels handed to a lambda that launches them
    return names | set(re.findall(r"\b(?:run|gradients)\((k_\w+)", text))


def test_every_early_kernel_is_found():
    assert {"k_bounds_partial", "k_sort_cells", "k_neighbours", "k_gradients", "k_timestep",
            "k_update"} <= launched_early() <= set(kernels())


@pytest.mark.parametrize("name", sorted(launched_early()))
def test_early_kernels_wait_first_and_promise_nothing(name):
    params, first = kernels()[name]
    assert first == "step_begin();"
    assert set(re.findall(r"__restrict__ (\w+)", params)) <= FIXED
