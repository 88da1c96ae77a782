"""All sweeps of a small grid in one cluster launch (csrc/jacobi_cluster.cu)
against the FP32 oracle, bit for bit: sides of a cell or two, odd rows (a pair
with one cell), fewer planes than blocks, planes that leave the last blocks
short or empty, the most pairs a block takes and one more (the other route),
and odd counts of sweeps (the result in the other buffer) over several steps."""
import numpy as np
import pytest

from vof_b200 import ic

pytestmark = pytest.mark.gpu

CASES = [(2, 2, 2, 4, 3), (3, 1, 5, 3, 4), (1, 1, 3, 10, 2), (1, 2, 40, 5, 3), (5, 4, 16, 10, 2), (6, 3, 17, 7, 3),
         (7, 6, 31, 4, 3), (24, 20, 16, 10, 3), (33, 15, 33, 3, 4), (32, 32, 32, 10, 3), (32, 32, 32, 6, 2),
         (31, 32, 32, 9, 3), (34, 32, 32, 10, 2), (64, 16, 30, 7, 3), (300, 6, 12, 5, 3), (9, 200, 15, 3, 3),
         (900, 1, 3, 4, 2)]


@pytest.mark.parametrize("nx,ny,nz,iters,steps", CASES)
def test_sweeps_bitwise_vs_oracle(cuda, V, orc, nx, ny, nz, iters, steps):
    prm = V.default_params(nx, ny, nz, dt=2e-4, gy=0.0, gz=-9.81, jacobi_iters=iters)
    state = ic.random_state(prm, seed=nx + 2 * ny + 3 * nz, vel_scale=0.5)
    rng = np.random.default_rng(nx)
    some = rng.random(state["p"].shape) < 0.1  # zeros, tiny and large values beside ordinary ones
    state["p"][some] = (rng.standard_normal(state["p"].shape) * 10.0 ** rng.uniform(-44, 9, state["p"].shape))[some]
    state["p"][rng.random(state["p"].shape) < 0.1] = 0.0
    with V.Solver(prm) as s:
        s.upload_state(**state)
        s.step(1)
        s.run(2, steps - 1)
        got = s.state()
    want = orc.run_f32(prm, state, 1, steps)
    for k in ("p", "u", "v", "w", "F"):
        # (NaN where the oracle has one: the large pressures overflow within four steps)
        assert np.array_equal(got[k], want[k], equal_nan=True), (k, int((got[k] != want[k]).sum()))
