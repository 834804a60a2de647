"""What the kernels' declarations promise the compiler, read from the sources:
a broken promise is a misaligned access or a stale read on the GPU, which no
test may provoke there.
"""
import re

import pytest

from conftest import REPO

CSRC = REPO / "rast-3dmhd-cpp_gb300" / "csrc"
SOURCES = sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh"))


def code(path):
    """The file without comments."""
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_dynamic_shared_memory_is_aligned_for_doubles(path):
    """Dynamic shared memory starts after a kernel's static shared data, at the
    alignment of its declaration and no more: a buffer in which doubles lie is
    declared as doubles or with that alignment."""
    for align, typ in re.findall(r"extern\s+__shared__\s+(__align__\(\d+\)\s+)?(\w[\w ]*?)\s*\w+\[\]", code(path)):
        n = int(re.search(r"\d+", align).group()) if align else {"double": 8, "double2": 16, "float4": 16}.get(typ, 4)
        assert n >= 8, f"{path.name}: {typ}"


def overlapped_kernels():
    """(file, kernel, declaration) of every kernel launched with launch_overlapped or waiting for the one before."""
    found = []
    for path in SOURCES:
        text = code(path)
        named = set(re.findall(r"launch_overlapped\(\s*(k_\w+)", text))
        heads = list(re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^{]*?\)\s+)?(k_\w+)\(([^{]*)\)\s*\{", text))
        for m, end in zip(heads, [h.start() for h in heads[1:]] + [len(text)]):
            if m.group(1) in named or "wait_previous()" in text[m.end():end]:
                found.append((path.name, m.group(1), m.group(2)))
    return found


def test_overlapped_kernels_promise_no_read_only_memory():
    """A kernel that starts while the one before it still writes may not declare
    what that one writes as const __restrict__: such loads may take the
    read-only path, which is defined for memory that nothing changes while the
    kernel runs, and need not stay behind the wait."""
    found = overlapped_kernels()
    assert {k for _, k, _ in found} >= {"k_substage", "k_substage_mixed", "k_bcon_ghost", "k_substage32",
                                       "k_bcon_ghost32", "k_flux", "k_cfl_seed", "k_cfl_rows"}
    for path, kernel, parameters in found:
        assert "__restrict__" not in parameters, (path, kernel)
