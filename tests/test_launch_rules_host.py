"""Order of the steps of chained kernels (csrc/common.cuh, chain_begin), read from the sources: a breach would show on a
GPU only as a rare hang or a stale read."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qs3_b200", "csrc")


def _kernels():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
            for part in src.split("__global__")[1:]:
                body = part.split("\n}\n")[0]
                yield pytest.param(body, id=f"{name}:{re.search(r'\b(\w+_kernel)\(', body)[1]}")


@pytest.mark.parametrize("body", list(_kernels()))
def test_tensor_memory_is_allocated_before_the_successor_is_released(body):
    release = [m.start() for m in re.finditer(r"chain_(begin|release)\(\)", body)]
    alloc = body.find("tcgen05.alloc")
    if alloc >= 0 and release:
        assert alloc < min(release)


def test_chained_kernels_wait_for_their_predecessor():
    bodies = {p.id.split(":")[1]: p.values[0] for p in _kernels()}
    chained = set()
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
            for m in re.finditer(r"launch_chained(?:_cluster)?\(([^;]*);", src):
                named = re.findall(r"\b\w+_kernel\b", m[1])
                # a local variable: the kernels assigned to it earlier in the same function
                scope = src[:m.start()].rsplit("\n}\n", 1)[-1]
                chained |= set(named or re.findall(r"\b\w+_kernel\b", "".join(re.findall(r"auto kernel = ([^;]*);", scope))))
    assert len(chained) > 15
    for kernel in chained:
        assert re.search(r"chain_(begin|wait)\(\)", bodies[kernel]), kernel
