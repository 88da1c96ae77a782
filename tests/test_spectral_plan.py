"""Which systems the direct pressure solve takes (csrc/spectral_plan.h): the
cyclic reduction along z ends well within its limit of steps on all of them, and
boxes so flat that a column's alpha rounds to 1/2 in FP64, where its recurrence
never ends, are left to the V-cycle and its bounded count.  On the host alone:
no such box is run."""
import ctypes as C
import os
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "cuda-lbm-ibm-fvm_b200" / "csrc"


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    lib = tmp_path_factory.mktemp("plan") / "libplan.so"
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    str(CSRC), str(HERE / "cpp" / "spectral_plan.cpp"), "-o", str(lib)], check=True)
    so = C.CDLL(str(lib))
    so.takes.argtypes = [C.c_int, C.c_int] + [C.c_float] * 3
    so.steps.argtypes = [C.c_double, C.c_double, C.c_int, C.c_int]
    so.least_ratio.restype = C.c_double
    return so


def box(V, plan, shape, **sides):
    p = V.default_params(*shape, **sides)
    return bool(plan.takes(p.nx, p.ny, p.dxi, p.dyi, p.dzi))


def test_the_reduction_ends_within_its_steps(plan):
    for e in np.linspace(np.log2(plan.least_ratio()), 60.0, 4001):
        for contracted in (0, 1):
            # (the kernel's limit is above the 27 or so steps of the least ratio by as many again)
            assert plan.steps(1.0, 2.0 ** e, contracted, 1000) <= plan.most_steps() - 15, e
    # below 2^-53 alpha is 1/2 and stays there
    assert plan.steps(1.0, 2.0 ** -54, 0, 1000) == 1000 and plan.steps(1.0, 2.0 ** -54, 1, 1000) == 1000


@pytest.mark.parametrize("shape,sides", [((200, 200, 200), {}), ((905, 905, 905), {}), ((905, 1, 905), {}),
                                         ((1, 1, 9000), {}), ((100, 80, 126), dict(Lx=0.3, Ly=0.1, Lz=0.05)),
                                         ((200, 200, 200), dict(Lx=1.0, Ly=1.0, Lz=0.001)),
                                         ((32, 32, 32), dict(Lz=1e6)), ((64, 64, 64), dict(Lx=1e-3, Ly=1e-3, Lz=10.0))])
def test_ordinary_boxes_are_taken(V, plan, shape, sides):
    assert box(V, plan, shape, **sides)


@pytest.mark.parametrize("shape,sides", [((32, 32, 32), dict(Lx=100.0, Ly=0.1, Lz=1e-6)),
                                         ((32, 32, 32), dict(Lx=1000.0, Ly=1000.0, Lz=1e-5)),
                                         ((200, 200, 200), dict(Lx=1e3, Ly=1e3, Lz=1e-3)),
                                         ((64, 64, 64), dict(Lx=np.inf)), ((64, 64, 64), dict(Ly=np.inf)),
                                         ((64, 64, 64), dict(Lz=np.inf)), ((64, 64, 64), dict(Lx=1e-44)),
                                         ((64, 64, 64), dict(Lz=1e-44))])
def test_boxes_whose_alpha_rounds_to_a_half_are_not(V, plan, shape, sides):
    with np.errstate(divide="ignore", over="ignore"):
        assert not box(V, plan, shape, **sides)
