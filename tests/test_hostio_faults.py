"""Staged copies (csrc/hostio.cu) when a CUDA call under them fails: the error comes back, and later copies neither wait for
chunks that were never sent nor deliver wrong bytes. Runs on the CPU against a stand-in for the runtime calls."""
import subprocess
from pathlib import Path

import pytest

from tensorlisp_b200 import build

HERE = Path(__file__).resolve().parent
WRAPPED = ("SetDevice HostAlloc FreeHost PointerGetAttributes GetLastError EventCreateWithFlags EventRecord EventSynchronize "
           "MemcpyAsync StreamSynchronize").split()


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = tmp_path_factory.mktemp("hostio") / "faults"
    cmd = [build._nvcc()] + build.ARCH + ["-O1", "-std=c++17", "-I", str(build.CSRC), "-o", str(exe), str(HERE / "hostio_faults.cpp"),
                                          str(build.CSRC / "hostio.cu")]
    for name in WRAPPED:
        cmd += ["-Xlinker", "--wrap=cuda" + name]
    build._run(cmd, False)
    return exe


# the first and second half ring, in the middle, the last chunk (41 chunks; a download first waits for the ring's 16 slots)
@pytest.mark.parametrize("what,at", [("d2h_wait", 0), ("d2h_wait", 16), ("d2h_wait", 30), ("d2h_wait", 56), ("d2h_copy", 0), ("d2h_copy", 9), ("d2h_copy", 40),
                                     ("h2d_copy", 0), ("h2d_copy", 17), ("h2d_copy", 40), ("h2d_wait", 0), ("h2d_wait", 24)])
def test_an_error_is_reported_and_the_ring_goes_on(program, what, at):
    r = subprocess.run([str(program), what, str(at)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("what", ["device_up", "device_down"])
def test_helper_threads_call_for_the_device_of_the_copy(program, what):
    r = subprocess.run([str(program), what], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


def test_results_that_are_kept_and_results_that_come_back(program):
    r = subprocess.run([str(program), "results"], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
