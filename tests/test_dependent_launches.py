"""The contract of the programmatic dependent launches (emergence_b200/csrc/
launch.cuh), checked on the sources: a kernel launched that way exists while the
one before it still writes, so it waits before it does anything else and loads
nothing through the read-only path, whose promise (no one writes this memory
while the kernel lives) it cannot keep. Tables uploaded before the launches
(block lists, levels, cell sizes) may be read-only."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "emergence_b200", "csrc")
SOURCES = {f: open(os.path.join(CSRC, f), encoding="utf-8").read()
           for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))}
UPLOADED = {"dxl"}  # floating-point tables that no kernel writes


def _close(text, i, pair):
    """Index behind the bracket that closes the one before i."""
    depth = 1
    while depth:
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        i += 1
    return i


def _kernels():
    """name -> (parameter list, body) of every __global__ definition."""
    found = {}
    for text in SOURCES.values():
        for m in re.finditer(r"__global__\s+(?:void\s+)?(\w+)\s*\(", text):
            name, i = m.group(1), m.end()
            if name == "__launch_bounds__":
                n = re.compile(r"\s*(?:void\s+)?(\w+)\s*\(").match(text, _close(text, i, "()"))
                name, i = n.group(1), n.end()
            j = _close(text, i, "()")
            body = re.compile(r"\s*\{").match(text, j)
            if body:
                found[name] = (text[i:j - 1], text[body.end():_close(text, body.end(), "{}") - 1])
    return found


KERNELS = _kernels()
DEPENDENT = sorted({m.group(2) for text in SOURCES.values()
                    for m in re.finditer(r"launch_dependent\(\s*((?:NVK|PHK)\()?(\w+)", text)} - {"void"})


def test_every_dependent_kernel_is_found():
    assert len(DEPENDENT) >= 20 and set(DEPENDENT) <= set(KERNELS), set(DEPENDENT) - set(KERNELS)


@pytest.mark.parametrize("name", DEPENDENT)
def test_waits_before_anything_else(name):
    body = KERNELS[name][1]
    sweep = re.match(r"\s*(?:Five)?Sweep<[^;]*>::run\(p\);\s*$", body)
    assert sweep or re.match(r"\s*dependency_wait\(\);", body), name


@pytest.mark.parametrize("file", ["sweep.cuh", "five_sweep.cuh"])
def test_sweeps_wait_before_they_read_the_control_block(file):
    run = SOURCES[file].split("static void run(", 1)[1]
    assert run.index("dependency_wait();") < run.index("->done")


@pytest.mark.parametrize("name", DEPENDENT)
def test_no_read_only_view_of_what_kernels_write(name):
    views = re.findall(r"const\s+double\s*\*\s*__restrict__\s+(\w+)", KERNELS[name][0])
    assert set(views) <= UPLOADED, (name, views)


@pytest.mark.parametrize("file", list(SOURCES))
def test_no_read_only_loads_of_the_state(file):
    text = SOURCES[file]
    assert "__ldg(" not in text and "ld.global.nc" not in text
    for m in re.finditer(r"struct (\w*Params) \{(.*?)\n\};", text, re.S):
        assert "__restrict__" not in m.group(2), m.group(1)
