"""Kernels launched with programmatic dependent launch (csrc/chain.cuh) are
resident while the kernel before them writes what they read. Loads through the
read-only path (__ldg, const __restrict__ kernel parameters) need memory that
nobody writes from the launch on, so the sources of such kernels have none for
the state, face-B and scratch arrays."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dragon_b200", "csrc")
KERNEL = re.compile(r"__global__[^;{]*?\b(k_\w+)\s*\(([^{;]*)\)\s*\{\s*(chained(?:_last)?\(\);)?", re.S)


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def kernels():
    return [(name, m.group(1), m.group(2), m.group(3)) for name in sorted(os.listdir(CSRC))
            if name.endswith((".cu", ".cuh")) for m in KERNEL.finditer(source(name))]


def test_chained_kernels_are_found_and_are_the_launched_ones():
    found = {k for _, k, _, c in kernels() if c}
    launched = {k for name in os.listdir(CSRC) if name.endswith((".cu", ".cuh"))
                for k in re.findall(r"chain\((k_\w+)", source(name))}
    assert len(found) > 20 and launched <= found, launched - found


@pytest.mark.parametrize("name,kernel,params", [k[:3] for k in kernels() if k[3]], ids=lambda v: str(v)[:24])
def test_no_read_only_loads(name, kernel, params):
    arrays = [p for p in params.split(",") if re.search(r"const\s+(double|float)\s*\*\s*__restrict__", p)]
    assert not arrays, arrays
    assert "__ldg" not in source(name)
