"""The direct pressure solve of the convergent modes (cosine transforms along x
and y, cyclic reduction along z; csrc/spectral.cu) at the sizes where its
tiling can go wrong: sides of 1, around the 16-row and 8-step matrix tiles, the
32-line blocks, the 8- and 16-warp launches (sides of 256 and 512), the
narrower blocks of long sides (over 704 along x or y, over 208 and 416 along
z), odd sides (a middle cell without a partner)."""
import numpy as np
import pytest

from vof_b200 import ic

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    a, b = a.astype(np.float64), b.astype(np.float64)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


SHAPES = [(1, 90, 100), (90, 1, 100), (100, 90, 1), (2, 65, 64), (33, 32, 17), (31, 16, 33), (32, 48, 15),
          (24, 26, 28), (17, 19, 41), (256, 6, 7), (257, 7, 6), (7, 258, 6), (6, 255, 7), (513, 5, 5), (5, 514, 5),
          (705, 4, 4), (4, 720, 4), (7, 6, 208), (6, 7, 209), (5, 5, 417), (4, 4, 801)]


@pytest.mark.parametrize("shape", SHAPES)
def test_direct_solve_vs_fp64_oracle(cuda, V, orc, shape):
    prm = V.default_params(*shape, dt=2e-4, mode=V.MODE_FP64, tol=1e-10, max_outer=3)
    state = ic.random_state(prm, seed=sum(shape), vel_scale=0.5)
    with V.Solver(prm) as s:
        s.upload_state(**state)
        s.step(1)
        stats = s.solver_stats()
        p = s.download("p")
    assert stats["outer"] <= 2 and stats["rel_final"] <= 1e-10, stats
    ref = orc.run_conv_f64(prm, state, 1, 1, tol=1e-12)
    inner = (slice(1, -1),) * 3
    # the two right-hand sides differ by FP32 rounding: u* to 2^-24, its divergence and the pressure to 1e-5
    assert rel_l2(p[inner], ref["p"][inner]) <= 1e-5


@pytest.mark.parametrize("mode", ["MODE_MIXED", "MODE_FP64"])
@pytest.mark.parametrize("shape", [(64, 64, 64), (30, 40, 35)])
def test_direct_solve_agrees_with_the_v_cycles(cuda, V, monkeypatch, mode, shape):
    """Both solve the same system to 1e-10 in FP64 residuals (the residual bounds
    the FP32 fields' difference far below 1e-6)."""
    prm = V.default_params(*shape, dt=2e-4, mode=getattr(V, mode), tol=1e-10, max_outer=100)
    state = ic.random_state(prm, seed=21, vel_scale=0.5)
    got = []
    for cycles in (False, True):
        if cycles:
            monkeypatch.setenv("VOF_MG_PAIRS", "1")
        with V.Solver(prm) as s:
            s.upload_state(**state)
            for n in (1, 2, 3):
                s.step(n)
            got.append((s.state(), s.solver_stats()))
    (direct, st), (cycled, sc) = got
    assert st["outer"] < sc["outer"] and st["rel_final"] <= 1e-10 and sc["rel_final"] <= 1e-10
    inner = (slice(1, -1),) * 3
    for k in ("F", "u", "v", "w", "p"):
        assert rel_l2(direct[k][inner], cycled[k][inner]) <= 1e-6, k


def test_a_start_value_that_meets_the_tolerance_is_left(cuda, V):
    """The pressure of a solve taken as the next one's start: the correction's
    kernels find the residual small on the device and leave the pressure."""
    prm = V.default_params(32, dt=2e-4, mode=V.MODE_FP64, tol=1e-6, max_outer=5)
    state = ic.random_state(prm, seed=4, vel_scale=0.3)
    state["p"][:] = 0.0
    with V.Solver(prm) as s:
        s.upload_state(**state)
        s.step(1)
        assert s.solver_stats()["outer"] == 1
        p = s.download("p")
    prm2 = V.default_params(32, dt=2e-4, mode=V.MODE_FP64, tol=1e-4, max_outer=5)
    with V.Solver(prm2) as s:
        s.upload_state(**dict(state, p=p))
        s.step(1)
        st = s.solver_stats()
        q = s.download("p")
    assert st["outer"] == 0 and st["rel_initial"] == st["rel_final"] <= 1e-4
    inner = (slice(1, -1),) * 3
    assert rel_l2(q[inner], p[inner]) <= 1e-6  # the gauge alone
