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
