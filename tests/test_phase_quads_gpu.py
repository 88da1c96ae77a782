"""The four-cell correction and right-hand side where quads of one phase, and of
any other equal value, take one density for all their faces: boxes of constant
F with values of either side of the clamp, bit for bit against the FP32 oracle,
at row lengths of every remainder of a quad.  The choice by size is forced
(VOF_CORRECT, VOF_RHS are read once per process: in a child)."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from vof_b200 import ic

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent
SHAPES = [(1, 2, 3), (2, 5, 1), (3, 1, 4), (4, 4, 4), (5, 9, 7), (30, 12, 6), (31, 7, 9), (32, 6, 5), (33, 20, 8),
          (126, 5, 4), (129, 4, 5)]
CODE = """
import sys, numpy as np
sys.path.insert(0, sys.argv[1])
import vof_b200 as V
for q in range(int(sys.argv[3])):
    f = np.load(f"{sys.argv[2]}/in{q}.npz")
    nx, ny, nz = (int(x) for x in f["case"])
    with V.Solver(V.default_params(nx, ny, nz, dt=2e-4, gy=0.0, gz=-9.81, jacobi_iters=4)) as s:
        s.upload_state(**{k: f[k] for k in "Fuvwp"})
        s.step(1)
        np.savez(f"{sys.argv[2]}/out{q}.npz", **s.state())
"""


def boxes(prm, seed):
    """F of constant boxes (pure, mixed, beyond the clamp, subnormal, of the other zero)."""
    rng = np.random.default_rng(seed)
    values = np.float32([0.0, 1.0, 0.37, 0.9999, -0.0, 1.25, -0.5, 1e-41, 1e-9])
    edges = [np.cumsum(rng.integers(1, 12, n)) for n in prm.shape]
    part = [np.searchsorted(e, np.arange(n), side="right") for e, n in zip(edges, prm.shape)]
    pick = rng.integers(0, len(values), [p.max() + 1 for p in part])
    return values[pick[np.ix_(*part)]]


def test_boxes_of_equal_F_bitwise_vs_oracle(cuda, V, orc, tmp_path):
    cases = []
    for q, shape in enumerate(SHAPES):
        prm = V.default_params(*shape, dt=2e-4, gy=0.0, gz=-9.81, jacobi_iters=4)
        state = dict(ic.random_state(prm, seed=q, vel_scale=0.5), F=boxes(prm, q))
        np.savez(tmp_path / f"in{q}.npz", case=shape, **state)
        cases.append((prm, state))
    subprocess.run([sys.executable, "-c", CODE, str(ROOT / "cuda-lbm-ibm-fvm_b200"), str(tmp_path), str(len(cases))],
                   env={**os.environ, "VOF_CORRECT": "4", "VOF_RHS": "4"}, check=True, timeout=600)
    for q, (prm, state) in enumerate(cases):
        got, want = dict(np.load(tmp_path / f"out{q}.npz")), orc.run_f32(prm, state, 1, 1)
        for k in ("p", "u", "v", "w", "F"):
            assert np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)), (SHAPES[q], k)
