"""What a kernel launched through overlapping() has to do, read from the sources (no device): in a captured step it becomes resident while the kernel in front still runs,
so it waits (after_previous) and reads memory on no path that is defined only for data nobody writes while it runs (ld.global.nc: ldg_stream, __ldg, const __restrict__)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "simplellminference_b200", "csrc")
READ_ONLY = re.compile(r"\bldg_stream8?\s*\(|\b__ldg\s*\(|global\.nc\b|__restrict__")


def _sources():
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        out[os.path.basename(path)] = text
    return out


def _kernels(text):
    """(name, parameters and body) of every kernel of a file."""
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
        brace = text.find("{", m.end())
        if brace < 0 or ";" in text[m.end():brace]:
            continue                       # a declaration
        depth, end = 1, brace + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        yield m.group(1), text[m.start():end]


WAITING = {name: (f, code) for f, text in _sources().items() for name, code in _kernels(text) if "after_previous()" in code}


def test_every_overlapping_launch_is_of_a_kernel_that_waits():
    launched = {n for f, text in _sources().items() if f != "common.cuh" for n in re.findall(r"overlapping(?:_alone)?\(\s*(\w+)", text)} - {"kernel"}     # `kernel`: a launcher's parameter
    assert len(launched) > 50 and launched <= set(WAITING), launched - set(WAITING)


@pytest.mark.parametrize("file", sorted({f for f, _ in WAITING.values()}))
def test_no_read_only_loads_in_files_of_kernels_that_wait(file):
    """The whole file: helpers of its kernels are in it."""
    found = READ_ONLY.search(_sources()[file])
    assert found is None, (file, found.group(0))
