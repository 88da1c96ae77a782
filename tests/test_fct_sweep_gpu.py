"""The FCT sweep kernels (csrc/fct_sweep.cu) against the FP32 oracle, bit for bit,
at the sizes where their tiles can go wrong: sides of one and two cells, lines
that fill a block of one position per thread exactly, by one more or less, or
are too long for it, tiles of 26 and 42 cells along a line, rows that fill a
tile once, twice or not quite, and states with gas (blocks of zeros), liquid
and interfaces in all three sweep orders."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 7), (7, 1, 2), (2, 9, 1), (30, 31, 32), (33, 62, 29), (61, 30, 63), (126, 15, 7), (15, 127, 9),
          (9, 13, 128), (254, 5, 6), (6, 255, 5), (5, 6, 256),  # one position per thread, or too long for it
          (26, 160, 140), (150, 27, 140), (150, 140, 52), (54, 104, 105), (104, 107, 130), (170, 79, 53),
          (254, 60, 60), (255, 52, 53), (340, 45, 44), (510, 40, 41), (620, 30, 31), (905, 25, 26)]  # tiles


def state_of(prm, seed):
    """Gas above a rough surface, liquid with some foam below, velocities of both signs."""
    rng = np.random.default_rng(seed)
    shape = prm.shape
    F = np.clip(rng.uniform(-0.4, 1.6, shape), 0, 1).astype(np.float32)
    z = np.arange(shape[0])[:, None, None] / shape[0]
    F = np.where(z > 0.45 + 0.1 * rng.random((1,) + shape[1:]), np.float32(0), F)
    vel = {k: (0.6 * rng.standard_normal(shape)).astype(np.float32) for k in "uvw"}
    return {"F": F, **vel, "p": rng.standard_normal(shape).astype(np.float32)}


def check(V, orc, shape, steps, **kw):
    prm = V.default_params(*shape, dt=2e-4, gy=0.0, gz=-9.81, **kw)
    state = state_of(prm, sum(shape))
    with V.Solver(prm) as s:
        s.upload_state(**state)
        s.run(1, steps)
        got = s.state()
    want = orc.run_f32(prm, state, 1, steps)
    for k in ("F", "u", "v", "w", "p"):
        assert np.array_equal(got[k], want[k]), (k, int((got[k] != want[k]).sum()))


@pytest.mark.parametrize("shape", SHAPES)
def test_sweeps_bitwise_vs_oracle(cuda, V, orc, shape):
    check(V, orc, shape, 3)  # all three sweep orders, each axis last once


def test_six_positions_per_thread(cuda, V, orc):
    """From 2^25 cells the y and z tiles hold 42 cells of a line."""
    check(V, orc, (900, 230, 170), 1, jacobi_iters=2)
