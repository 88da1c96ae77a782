"""The threaded device to host copy (csrc/host_pull.cu) on the host, over a fake
of the runtime calls that it makes: whatever a thread's start fails with (no
thread to be had, no memory for its state), the other threads are joined, their
slices copied and no exception leaves the call."""
import os
import subprocess
from pathlib import Path

from vof_b200 import build

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "cuda-lbm-ibm-fvm_b200" / "csrc"


def test_copies_are_whole_whatever_a_thread_start_fails_with(tmp_path):
    exe = tmp_path / "host_pull"
    subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-pthread", "-Wl,--wrap=pthread_create",
                    "-static-libstdc++", "-I", str(CSRC), "-I", str(build.cuda_home() / "include"),
                    str(HERE / "cpp" / "host_pull.cpp"), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, (run.returncode, run.stdout, run.stderr)
