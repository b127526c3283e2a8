"""Scalars read back from the device."""
import subprocess

import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu


def test_announcement_ends_with_its_scope(lib_path, tmp_path):
    """After an exception between the announcement of a norm and its fetch, later fetches of that scalar return its
    present value (the announcement is internal to the library: a program against its headers)."""
    import build
    exe = tmp_path / "announced_fetch"
    r = subprocess.run([build.nvcc(), *build.NVCC_FLAGS, f"-I{build.CSRC}", str(ROOT / "tests" / "cpp" / "announced_fetch.cu"),
                        "-o", str(exe), f"-L{PKG}", "-lnuma_gpu", "-Xlinker", f"-rpath={PKG}"], text=True, capture_output=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], text=True, capture_output=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    assert [float(v) for v in out.stdout.split()] == [2.0, 3.0, 4.0]
