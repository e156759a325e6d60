"""Kernels that may be set up while the one before them drains wait for it first."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "stardust_b200" / "csrc"
SOURCES = [p for p in sorted(CSRC.glob("*.cu")) if re.search(r"\blaunch\(", p.read_text())]


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_every_overlapped_kernel_waits_first(path):
    """launch() lets a kernel begin before its predecessor's writes can be seen, so the first
    statement of each kernel in such a file is the wait, unless it is launched plainly only."""
    src = path.read_text()
    plain = set(re.findall(r"\b(k_\w+)(?:<[^;()]*?>)?<<<", src))
    kernels = re.findall(r"__global__[^;{]*?\b(k_\w+)\s*\([^{]*\{\s*(\w+)", src)
    assert len(kernels) == len(re.findall(r"__global__", src))
    for name, first in kernels:
        assert first == "wait_previous" or name in plain, name
    for name in plain:
        assert f"launch({name}" not in src
