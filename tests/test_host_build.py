"""The native host path is built where it is missing or does not fit, once, whole, and not at import."""

import os
import pathlib
import shutil
import stat
import subprocess
import sys

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]


@pytest.fixture()
def copy(tmp_path):
    """A checkout of the package without the host path, and a g++ that takes a second, notes its run and
    leaves the module that is built here."""
    from mosaicist_b200 import build

    build.build_host_ops()
    pkg = tmp_path / "mosaicist_b200"
    shutil.copytree(ROOT / "mosaicist_b200", pkg, ignore=shutil.ignore_patterns("_host_ops.*", "__pycache__"))
    shutil.copytree(ROOT / "include", tmp_path / "include")
    tools = tmp_path / "bin"
    tools.mkdir()
    gxx = tools / "g++"
    gxx.write_text(f"""#!{sys.executable}
import shutil, sys, time
out = sys.argv[sys.argv.index("-o") + 1]
with open({str(tmp_path / "runs")!r}, "a") as f:
    f.write("run\\n")
data = open({str(build.HOST_OPS)!r}, "rb").read()
with open(out, "wb") as f:                     # a part, then the rest
    f.write(data[:4096]); f.flush(); time.sleep(1.0); f.write(data[4096:])
""")
    gxx.chmod(gxx.stat().st_mode | stat.S_IEXEC)
    return tmp_path


def _start(copy, code, with_gxx=True):
    env = dict(os.environ, PATH=str(copy / "bin") if with_gxx else str(copy / "none"), PYTHONPATH=str(copy))
    return subprocess.Popen([sys.executable, "-c", code], cwd=copy, env=env, stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True)


def _done(*procs):
    for p in procs:
        out, err = p.communicate(timeout=240)
        assert p.returncode == 0, err
    return out, err


def test_import_and_tracing_need_no_compiler(copy):
    out, err = _done(_start(copy, """
import mosaicist_b200.ops, mosaicist_b200.moe, mosaicist_b200.parallel
import mosaicist_b200.torch_ops as t, torch, importlib
from torch._subclasses.fake_tensor import FakeTensorMode
def trace():
    with FakeTensorMode():
        a, b = (torch.empty(s, dtype=torch.bfloat16, device="cuda") for s in ((64, 128), (128, 256)))
        return tuple(torch.ops.mosaicist_sm100a.gemm_f16(a, b).shape)
assert trace() == (64, 256)
importlib.reload(t)
assert trace() == (64, 256)
try:
    mosaicist_b200.ops.gemm_f16(torch.empty(8, 8), torch.empty(8, 8))
except RuntimeError as e:
    print(e)
""", with_gxx=False))
    assert "g++ not found" in out and "can be traced but not run" in err
    assert not (copy / "runs").exists() and not (copy / "mosaicist_b200" / "_host_ops.so").exists()


def test_processes_that_start_together_build_once(copy):
    code = "from mosaicist_b200 import _lib; assert callable(_lib.native.gemm_f16)"
    _done(*[_start(copy, code) for _ in range(4)])
    assert (copy / "runs").read_text().count("run") == 1
    assert not list((copy / "mosaicist_b200").glob("*.part"))
    _done(_start(copy, code, with_gxx=False))                  # what is there fits: no compiler needed
    stamp = copy / "mosaicist_b200" / "_host_ops.stamp"
    stamp.write_text(stamp.read_text().replace("torch ", "torch 0.0+"))
    _done(_start(copy, code))                                  # built for another torch: again
    assert (copy / "runs").read_text().count("run") == 2
    header = copy / "include" / "mosaicist_sm100a.h"
    header.write_text(header.read_text() + "/* a comment */\n")
    _done(_start(copy, code, with_gxx=False))
    header.write_text(header.read_text() + "int msc_another(void);\n")
    p = _start(copy, code, with_gxx=False)
    assert "g++ not found" in p.communicate(timeout=240)[1] and p.returncode != 0


def test_library_and_host_path_must_be_of_one_header(copy):
    from mosaicist_b200 import _lib, build

    assert _lib.load().msc_abi().decode() == build.abi()
    out, _ = _done(_start(copy, """
import ctypes, torch
from mosaicist_b200 import _lib, ops
from torch._subclasses.fake_tensor import FakeTensorMode
other = ctypes.CFUNCTYPE(ctypes.c_char_p)(lambda: b"another header")
fetch = _lib.addresses
_lib.addresses = lambda: dict(fetch(), msc_abi=ctypes.cast(other, ctypes.c_void_p).value)
with FakeTensorMode():
    a, b, c = (torch.empty(s, dtype=torch.bfloat16, device="cuda") for s in ((64, 128), (128, 64), (64, 64)))
try:
    ops.gemm_f16(a, b, out=c)
except RuntimeError as e:
    print(e)
"""))
    assert "different headers" in out
