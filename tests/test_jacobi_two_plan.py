"""The tiling of the two-sweep Jacobi launch (csrc/jacobi_two_plan.h): within the
limits of a TMA box (256 elements a side), of a block and of the launch on every
grid the library takes, two-dimensional ones among them; and such grids on a
GPU, bit for bit against the FP32 oracle."""
import ctypes as C
import os
import subprocess
from pathlib import Path

import numpy as np
import pytest

from vof_b200 import ic

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "cuda-lbm-ibm-fvm_b200" / "csrc"
MOST = 905  # the longest side vof_create takes


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    lib = tmp_path_factory.mktemp("plan") / "libplan.so"
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(CSRC),
                    str(HERE / "cpp" / "jacobi_two_plan.cpp"), "-o", str(lib)], check=True)
    return C.CDLL(str(lib))


@pytest.mark.parametrize("first,last,step", [((1, 1, 1), (70, MOST, MOST), (1, 8, 113)),
                                             ((1, 240, 1), (9, 520, MOST), (1, 1, 64)),
                                             ((71, 1, 1), (MOST, MOST, MOST), (6, 61, 301)),
                                             ((1, MOST, MOST), (MOST, MOST, MOST), (1, 1, 1)),
                                             ((1, 1, 1), (40, 40, 40), (1, 1, 1))])
def test_tilings_stay_within_the_limits_of_a_launch(plans, first, last, step):
    triple, bad = C.c_int * 3, (C.c_int * 3)()
    broken = plans.check_plans(triple(*first), triple(*last), triple(*step), bad)
    assert broken == 0, (broken, tuple(bad))


@pytest.mark.parametrize("shape,iters,forced,want", [((24, 20, 16), 10, 0, 0), ((64, 64, 64), 10, 0, 0),
                                                     ((80, 80, 80), 10, 0, 0), ((81, 81, 81), 10, 0, 1),
                                                     ((128, 64, 64), 10, 0, 1), ((905, 905, 905), 10, 0, 1),
                                                     ((200, 200, 200), 2, 0, 0), ((200, 200, 200), 3, 0, 1),
                                                     ((200, 200, 200), 10, 1, 0), ((6, 5, 4), 10, 2, 1),
                                                     ((6, 5, 4), 2, 2, 0), ((200, 200, 200), 0, 2, 0)])
def test_tables_are_made_where_two_sweeps_run(plans, shape, iters, forced, want):
    """Only these calls set up the two-sweep launch: a step of a small grid in
    caller's memory does so on every call, for nothing otherwise."""
    assert plans.chosen(*shape, iters, forced) == want


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 512, 512), (2, 256, 256), (3, 253, 905), (1, 800, 800), (2, 700, 400)])
def test_two_dimensional_grids_bitwise_vs_oracle(cuda, V, orc, shape):
    prm = V.default_params(*shape, dt=2e-4, gy=0.0, gz=-9.81, jacobi_iters=4)
    state = ic.random_state(prm, seed=sum(shape), vel_scale=0.5)
    with V.Solver(prm) as s:
        s.upload_state(**state)
        s.step(1)
        got = s.state()
    want = orc.run_f32(prm, state, 1, 1)
    for k in ("p", "u", "v", "w", "F"):
        assert np.array_equal(got[k], want[k]), (k, int((got[k] != want[k]).sum()))
