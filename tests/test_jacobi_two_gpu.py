"""Two Jacobi sweeps per launch (csrc/jacobi_two.cu) against the FP32 oracle, bit
for bit, at the sizes where its tiles can go wrong: sides of a few cells, row
lengths at every remainder of a quad and either side of a second column of
tiles, rows and planes around a block's, odd counts of sweeps (one single sweep
first, the scratch buffer) and every buffer the result can land in.  The
choice by size is forced (VOF_JACOBI=two is read once per process: in a child)."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from vof_b200 import ic

pytestmark = pytest.mark.gpu

SHAPES = [(2, 2, 2, 4), (3, 1, 5, 3), (1, 1, 3, 10), (4, 5, 1, 6), (5, 4, 2, 5), (6, 3, 3, 4), (7, 6, 4, 7),
          (33, 30, 9, 4), (34, 31, 10, 3), (35, 32, 11, 5), (36, 33, 12, 6), (61, 29, 30, 4), (66, 28, 31, 10),
          (127, 13, 8, 4), (128, 14, 9, 3), (251, 7, 6, 4), (252, 6, 7, 5), (255, 5, 8, 4), (260, 34, 5, 4),
          (21, 150, 6, 4), (20, 9, 160, 4)]


ROOT = Path(__file__).resolve().parent.parent
CODE = """
import sys, numpy as np
sys.path.insert(0, sys.argv[1])
import vof_b200 as V
for q in range(int(sys.argv[3])):
    f = np.load(f"{sys.argv[2]}/in{q}.npz")
    nx, ny, nz, iters, steps = (int(x) for x in f["case"])
    prm = V.default_params(nx, ny, nz, dt=2e-4, gy=0.0, gz=-9.81, jacobi_iters=iters)
    with V.Solver(prm) as s:
        s.upload_state(**{k: f[k] for k in "Fuvwp"})
        for n in range(steps):
            s.step(1 + n)
        np.savez(f"{sys.argv[2]}/out{q}.npz", **s.state())
"""


def run_two(tmp_path, V, cases):
    """The states after each case's steps, every pair of sweeps in one launch."""
    for q, (prm, state, steps) in enumerate(cases):
        np.savez(tmp_path / f"in{q}.npz", case=[prm.nx, prm.ny, prm.nz, prm.jacobi_iters, steps], **state)
    subprocess.run([sys.executable, "-c", CODE, str(ROOT / "cuda-lbm-ibm-fvm_b200"), str(tmp_path), str(len(cases))],
                   env={**os.environ, "VOF_JACOBI": "two"}, check=True, timeout=600)
    return [dict(np.load(tmp_path / f"out{q}.npz")) for q in range(len(cases))]


def params(V, nx, ny, nz, iters):
    return V.default_params(nx, ny, nz, dt=2e-4, gy=0.0, gz=-9.81, jacobi_iters=iters)


def test_two_sweeps_bitwise_vs_oracle(cuda, V, orc, tmp_path):
    cases = []
    for nx, ny, nz, iters in SHAPES:
        prm = params(V, nx, ny, nz, iters)
        cases.append((prm, ic.random_state(prm, seed=nx + 2 * ny + 3 * nz, vel_scale=0.5), 3))
    for (prm, state, steps), got in zip(cases, run_two(tmp_path, V, cases)):
        want = orc.run_f32(prm, state, 1, steps)
        for k in ("p", "u", "v", "w", "F"):
            assert np.array_equal(got[k], want[k]), ((prm.nx, prm.ny, prm.nz), k, int((got[k] != want[k]).sum()))


def test_zero_tiny_and_large_pressures(cuda, V, orc, tmp_path):
    """Numerators outside the fast division's range beside ordinary ones in the
    same quads: exact zeros, values to the subnormal range, up to 1e30."""
    cases = []
    for shape in ((40, 36, 20), (13, 70, 9)):
        prm = params(V, *shape, 6)
        state = ic.rest_state(prm, ic.dam_break(prm))
        rng = np.random.default_rng(5)
        p = np.zeros(prm.shape, dtype=np.float32)
        m = rng.random(p.shape) < 0.3
        p[m] = (rng.standard_normal(p.shape) * 10.0 ** rng.uniform(-44, 10, p.shape)).astype(np.float32)[m]
        p[shape[2] // 2, shape[1] // 2, shape[0] // 2] = 1e30
        cases.append((prm, dict(state, p=p), 1))
    for (prm, state, steps), got in zip(cases, run_two(tmp_path, V, cases)):
        want = orc.run_f32(prm, state, 1, steps)["p"]
        assert np.isfinite(want).all()
        assert np.array_equal(got["p"], want), int((got["p"] != want).sum())
