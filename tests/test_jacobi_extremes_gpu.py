"""The three Jacobi kernels (one sweep per launch, two, all in a cluster) at the
ends of the FP32 range, bit for bit against the FP32 oracle: quotients beyond
the fast division's range in the cells, and ghost cells whose values enter only
through zero coefficients but would overflow in any arithmetic of their own.
The choice by size is forced (VOF_JACOBI is read once per process: in a child;
without it these grids take the cluster)."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from vof_b200 import ic

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent
SHAPES = [(12, 10, 9, 10), (7, 11, 6, 4), (26, 9, 12, 7), (33, 14, 10, 5), (30, 20, 8, 3)]
CODE = """
import sys, numpy as np
sys.path.insert(0, sys.argv[1])
import vof_b200 as V
for q in range(int(sys.argv[3])):
    f = np.load(f"{sys.argv[2]}/in{q}.npz")
    nx, ny, nz, iters = (int(x) for x in f["case"])
    with V.Solver(V.default_params(nx, ny, nz, dt=2e-4, gy=0.0, gz=-9.81, jacobi_iters=iters)) as s:
        s.upload_state(**{k: f[k] for k in "Fuvwp"})
        if "rhs" in f:
            s.upload("rhs", f["rhs"])
        s.step(1)
        np.savez(f"{sys.argv[2]}/out{q}.npz", **s.state())
"""


def step(tmp_path, env, cases):
    for q, (prm, fields) in enumerate(cases):
        np.savez(tmp_path / f"in{q}.npz", case=[prm.nx, prm.ny, prm.nz, prm.jacobi_iters], **fields)
    subprocess.run([sys.executable, "-c", CODE, str(ROOT / "cuda-lbm-ibm-fvm_b200"), str(tmp_path), str(len(cases))],
                   env={**os.environ, **env}, check=True, timeout=600)
    return [dict(np.load(tmp_path / f"out{q}.npz")) for q in range(len(cases))]


def params(V, nx, ny, nz, iters):
    return V.default_params(nx, ny, nz, dt=2e-4, gy=0.0, gz=-9.81, jacobi_iters=iters)


KERNELS = pytest.mark.parametrize("env", [{}, {"VOF_JACOBI": "peel"}, {"VOF_JACOBI": "two"}])


@KERNELS
def test_quotients_beyond_the_fast_division(cuda, V, orc, tmp_path, env):
    cases = []
    for shape in SHAPES:
        prm = params(V, *shape)
        state = ic.random_state(prm, seed=sum(shape), vel_scale=1.0)
        rng = np.random.default_rng(sum(shape))
        at = tuple(rng.integers(1, n - 1, 40) for n in prm.shape)
        state["p"][at] = (rng.standard_normal(40) * 1e31).astype(np.float32)
        state["p"][tuple(a[0] for a in at)] = 3.0e33
        cases.append((prm, state))
    for (prm, state), got in zip(cases, step(tmp_path, env, cases)):
        want = orc.run_f32(prm, state, 1, 1)
        assert np.isfinite(want["p"]).all() and np.abs(want["p"]).max() > 1e24
        for k in ("p", "u", "v", "w", "F"):  # (NaN where the correction of such pressures has one)
            assert np.array_equal(got[k], want[k], equal_nan=True), (prm.shape, k)


@KERNELS
def test_ghosts_that_would_overflow(cuda, V, orc, tmp_path, env):
    cases = []
    for shape in SHAPES:
        prm = params(V, *shape)
        state = ic.random_state(prm, seed=sum(shape), vel_scale=0.5)
        rng = np.random.default_rng(sum(shape))
        ghost = np.ones(prm.shape, dtype=bool)
        ghost[1:-1, 1:-1, 1:-1] = False
        state["p"][ghost] = (rng.choice([-1.0, 1.0], prm.shape) * 10.0 ** rng.uniform(30, 38, prm.shape))[ghost]
        rhs = np.zeros(prm.shape, dtype=np.float32)
        rhs[ghost] = rng.choice([np.nan, np.inf, -np.inf], prm.shape)[ghost]
        cases.append((prm, dict(state, rhs=rhs)))
    for (prm, fields), got in zip(cases, step(tmp_path, env, cases)):
        want = orc.run_f32(prm, {k: fields[k] for k in "Fuvwp"}, 1, 1)
        assert np.isfinite(want["p"][1:-1, 1:-1, 1:-1]).all()
        for k in ("p", "u", "v", "w", "F"):
            assert np.array_equal(got[k], want[k]), (prm.shape, k, int((got[k] != want[k]).sum()))
