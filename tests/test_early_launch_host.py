"""Kernels that are launched early (griddepcontrol) are resident while the kernel before
them still writes, so none of their loads may take the read-only path, whose data has to
be read-only for the whole life of the kernel: no __ldg, no ld.global.nc, and no
const __restrict__ pointer, from which the compiler makes such loads by itself."""
import re
from pathlib import Path

import pytest

SRC = Path(__file__).resolve().parent.parent / "compchan3dmpi_b200" / "csrc"


def code(path):
    s = re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", s)


@pytest.mark.parametrize("name", sorted(p.name for p in SRC.iterdir() if p.suffix in (".cu", ".cuh", ".h")))
def test_no_read_only_path_loads(name):
    found = re.findall(r"\b__ldg\b|\bld\.global(?:\.\w+)*\.nc\b|\b__restrict__\b", code(SRC / name))
    assert not found, found
