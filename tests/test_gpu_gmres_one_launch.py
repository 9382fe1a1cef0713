"""The one-launch GMRES solve (csrc/gmres_grid.cuh) at the edges of its launch
shapes: boxes of as many nodes as each worker count reaches and one row more,
a reduced axis, several restart cycles, a wall box, and columns past the limit
of its shared-memory triangles (the kernel-per-operation form).  Needs a GB300."""
import numpy as np
import pytest

import pyoracle as O
from picpp_gb300 import initstate as I

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pg():
    import picpp_gb300 as P
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    P.load_library()
    return P


def system(n, seed):
    rng = np.random.default_rng(seed)
    N = n[0] * n[1] * n[2]
    mu = 0.02 * rng.standard_normal((9, N))
    for d in (0, 4, 8):
        mu[d] -= 0.2
    return mu.reshape(-1), rng.standard_normal(3 * N)


def solve(pg, n, opts, seed, wall=False):
    box = I.Box(*n, 0.5, 0.45, 0.6, 0.5)
    kw = dict(boundary_x=pg.BOUNDARY_WALL_OPEN) if wall else {}
    sim = pg.GpuSimulation(box, pg.IMPLICIT, particle_real=1, pressure_compat=0, tile=(0, 0, 0), **kw)
    mu, rhs = system(n, seed)
    x, info = sim.maxwell_solve(mu, rhs, opts)
    sim.close()
    g = O.make_grid(box, pressure_compat=0, wall_x=1 if wall else 0)
    return g, mu, rhs, x, info


# 4,096, 24,576, 393,216 and 786,432 nodes, and a row more
@pytest.mark.parametrize("n", [(3, 1, 1), (16, 16, 16), (17, 16, 16), (32, 32, 24), (33, 32, 24), (96, 64, 64),
                               (97, 64, 64), (128, 96, 64), (129, 96, 64)])
def test_restarted_reaches_the_true_residual(pg, n):
    g, mu, rhs, x, info = solve(pg, n, pg.solve_opts(pg.GMRES_RESTARTED, restart=30, max_iter=200, tol=1e-9), 3)
    res = np.linalg.norm(O.maxwell_apply(g, mu, x) - rhs) / np.linalg.norm(rhs)
    # the device's true residual, evaluated again: rounding of one apply, far below 1e-12
    assert res <= 1e-9 + 1e-12
    assert abs(res - info["rel_residual"]) <= 1e-12


@pytest.mark.parametrize("restart,wall", [(1, False), (4, False), (128, False), (129, False), (10, True), (128, True),
                                          (129, True)])
def test_restart_lengths_and_walls(pg, restart, wall):
    g, mu, rhs, x, info = solve(pg, (12, 10, 6), pg.solve_opts(pg.GMRES_RESTARTED, restart=restart, max_iter=400, tol=1e-10),
                                4, wall)
    res = np.linalg.norm(O.maxwell_apply(g, mu, x) - rhs) / np.linalg.norm(rhs)
    assert res <= 1e-10 + 1e-13
    assert info["restarts"] >= (info["iterations"] + restart - 1) // restart


# a solve that stops at |r| / |b| <= 1e-8 / (3N) (or 1e-15) is within the operator's
# condition number (below 10 here) times that of the oracle's own
@pytest.mark.parametrize("n", [(16, 1, 1), (13, 11, 1), (16, 16, 16), (17, 16, 16), (33, 32, 24)])
@pytest.mark.parametrize("max_iter", [50, 130, 131])
def test_reference_method_matches_the_oracle(pg, n, max_iter):
    g, mu, rhs, x, info = solve(pg, n, pg.solve_opts(pg.GMRES_REFERENCE, max_iter=max_iter, tol=1e-8), 5)
    xo, its, rel = O.gmres(O.make_grid(I.Box(*n, 0.5, 0.45, 0.6, 0.5), pressure_compat=0, gmres_max_iter=max_iter), mu, rhs)
    bound = 20 * max(1e-8 / (3 * n[0] * n[1] * n[2]), 1e-15) + 1e-13
    assert np.linalg.norm(x - xo) <= bound * np.linalg.norm(xo)
    assert abs(info["iterations"] - its) <= 1


def test_non_finite_system_is_refused(pg):
    box = I.Box(8, 8, 8, 0.5, 0.5, 0.5, 0.5)
    sim = pg.GpuSimulation(box, pg.IMPLICIT, particle_real=1, pressure_compat=0)
    for bad in ("mu", "rhs"):
        mu, rhs = system((8, 8, 8), 6)
        (mu if bad == "mu" else rhs)[777] = np.inf
        with pytest.raises(pg.PicError, match="non-finite"):
            sim.maxwell_solve(mu, rhs, pg.solve_opts(pg.GMRES_RESTARTED))
    x, info = sim.maxwell_solve(*system((8, 8, 8), 6), pg.solve_opts(pg.GMRES_RESTARTED, tol=1e-8, max_iter=100))
    assert info["rel_residual"] <= 1e-8
    x, info = sim.maxwell_solve(system((8, 8, 8), 6)[0], np.zeros(3 * 512), pg.solve_opts(pg.GMRES_RESTARTED))
    assert not x.any() and info["iterations"] == 0
