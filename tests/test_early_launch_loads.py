"""Kernels that are set up under the launch before them (they call grid_dependency_wait) read what
that launch writes.  Such loads must be ordinary ones: data read with __ldg or ld.global.nc has to be
read-only for the kernel's whole life, and const __restrict__ inputs let the compiler choose that
form by itself.  A property of the source, so it is checked there."""

import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "mosaicist_b200" / "csrc"
READ_ONLY = re.compile(r"__ldg\s*\(|ld\.global\.nc|const\s+[\w:]+\s*\*\s*__restrict__")


def _functions(text):
    """Pieces of a file, one per function at namespace scope (a line that is '}' ends one)."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    return re.split(r"^\}[^\n]*$", text, flags=re.M)


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu*")), ids=lambda p: p.name)
def test_early_launched_kernels_use_ordinary_loads(path):
    for body in _functions(path.read_text()):
        if "grid_dependency_wait()" in body and "griddepcontrol" not in body:
            assert not READ_ONLY.search(body), READ_ONLY.search(body).group(0)


@pytest.mark.parametrize("name", ["gemm_common.cuh", "quantize_common.cuh", "quantize_rows.cuh"])
def test_what_those_kernels_share_uses_ordinary_loads(name):
    text = (CSRC / name).read_text()
    assert not READ_ONLY.search(text)


def test_the_check_sees_every_such_kernel():
    early = [p.name for p in CSRC.glob("*.cu*") if "grid_dependency_wait();" in p.read_text()]
    assert len(early) >= 9
