"""Scalars read back from the device."""
import subprocess

import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu


def _program(name, tmp_path):
    import build
    exe = tmp_path / name
    r = subprocess.run([build.nvcc(), *build.NVCC_FLAGS, f"-I{build.CSRC}", str(ROOT / "tests" / "cpp" / f"{name}.cu"),
                        "-o", str(exe), f"-L{PKG}", "-lnuma_gpu", "-Xlinker", f"-rpath={PKG}"], text=True, capture_output=True)
    assert r.returncode == 0, r.stderr
    return exe


def _run(exe, *args):
    out = subprocess.run([str(exe), *args], text=True, capture_output=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    return [float(v) for v in out.stdout.split()]


def test_announcement_ends_with_its_scope(lib_path, tmp_path):
    """After an exception between the announcement of a norm and its fetch, later fetches of that scalar return its
    present value (the announcement is internal to the library: a program against its headers)."""
    assert _run(_program("announced_fetch", tmp_path)) == [2.0, 3.0, 4.0]


def test_scalar_calls_leave_the_stream_idle(lib_path, tmp_path):
    """Calls that return a scalar synchronise the context's stream: 2,000 each of a norm, an inner product and a
    residual norm leave no work on it."""
    assert _run(_program("scalar_calls", tmp_path), "idle") == [0, 0, 0]


def test_waits_follow_the_device_schedule(lib_path, tmp_path):
    """Where the program has the device block its waiting threads (cudaDeviceScheduleBlockingSync), a wait of
    milliseconds for a norm leaves the core to others."""
    share, wall = _run(_program("scalar_calls", tmp_path), "blocking")
    assert wall > 2e-3 and share < 0.5
