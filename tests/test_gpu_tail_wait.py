"""A wait of the cluster kernel (k_tail.cu) that runs out: tests/cpp/tail_wait.cu, built
against the library's own launchers. No GPU fault is made: the wait's barrier expects
bytes that nothing sends, the wait gives up, and the kernel returns."""
import os
import subprocess

import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu


def test_tables_that_never_arrive(ctlib, ct, tmp_path):
    import build as build_module
    exe, libdir = str(tmp_path / "tail_wait"), os.path.dirname(ct.LIB_PATH)
    r = subprocess.run([build_module.nvcc(), *build_module.ARCH, "-std=c++17", "-I", os.path.join(PKG, "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "tail_wait.cu"), "-L", libdir, "-lcthermal",
                        f"-Xlinker=-rpath,{libdir}", "-o", exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    lines = [tuple(map(int, l.split()[1:])) for l in r.stdout.splitlines()]
    assert len(lines) == 6 and lines[0][0] > 1 and lines[2][0] > 1 and lines[4][0] == 1
    for late, good in zip(lines[::2], lines[1::2]):
        assert late[1:] == (1, 1, 1, 0)  # err, breakdown and done set, x untouched
        assert good[1:] == (0, 0, 0, 1)
