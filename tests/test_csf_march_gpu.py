"""The curvature's march and the accelerations in the predictor, against the
step-by-step restatement (tests/csf_model.py) bit for bit: grids at the edges of
the 30 x 14 column tiles and of the chunks of planes, F of droplets, of noise
and of boxes of equal values (the paths without a root or a quotient)."""
import numpy as np
import pytest

from csf_model import csf_increments, droplet
from vof_b200 import ic

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (1, 2, 3), (2, 1, 2), (30, 14, 5), (31, 15, 6), (29, 13, 1), (60, 28, 33), (61, 29, 2), (7, 43, 40),
          (64, 5, 130)]


@pytest.mark.parametrize("kind", ["droplet", "noise", "boxes"])
@pytest.mark.parametrize("shape", SHAPES)
def test_increments_bitwise(cuda, V, shape, kind):
    prm = [V.default_params(*shape, dt=1e-4, gy=0.0, gz=-9.81, surface_tension=q, sigma=0.07) for q in (0, 1)]
    rng = np.random.default_rng(sum(shape))
    if kind == "droplet":
        F = droplet(prm[0], R_cells=max(1.0, min(shape) / 3.0))
    elif kind == "noise":
        F = rng.random(prm[0].shape).astype(np.float32)
    else:
        F = np.kron(rng.integers(0, 3, [-(-n // 4) for n in prm[0].shape]), np.ones((4, 4, 4)))
        F = np.float32([0.0, 1.0, 0.99999])[F[tuple(slice(0, n) for n in prm[0].shape)].astype(int)]
    state = ic.rest_state(prm[0], F)
    for k in ("u", "v", "w"):
        state[k] = (0.01 * rng.standard_normal(prm[0].shape)).astype(np.float32)
    got = []
    for p in prm:
        with V.Solver(p) as s:
            s.upload_state(**state)
            s.step(1)
            got.append({k: s.download(k) for k in ("ustar", "vstar", "wstar")})
    for name, (d, mask) in zip(("ustar", "vstar", "wstar"), csf_increments(prm[1], F)):
        want = np.where(mask, got[0][name] + d, got[0][name]).astype(np.float32)
        bad = np.argwhere(got[1][name].view(np.uint32) != want.view(np.uint32))
        assert bad.size == 0, (name, len(bad), bad[:3])
