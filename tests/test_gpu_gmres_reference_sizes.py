"""The reference method of the one-launch GMRES solve (csrc/gmres_grid.cuh) at the
widths that only large boxes take, and in a wall box.  Needs a GB300."""
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


# 393,216 and 786,432 nodes are the last ones of 480 and of 736 workers a CTA
@pytest.mark.parametrize("n,wall", [((96, 64, 64), False), ((97, 64, 64), False), ((128, 96, 64), False),
                                    ((129, 96, 64), False), ((14, 10, 6), True), ((34, 32, 24), True),
                                    ((129, 96, 64), True)])
@pytest.mark.parametrize("max_iter", [12, 50])
def test_reference_reaches_the_residual_it_reports(pg, n, wall, max_iter):
    """50 columns take a system this well conditioned (about a factor of four a column) to
    the method's stop, |r| / |b| <= max(1e-8 / 3N, 1e-15) in exact arithmetic, of which
    rounding leaves some 1e-15 times the operator's norm (below 10); 12 columns
    leave it at the estimate, which then is the true residual but for that."""
    box = I.Box(*n, 0.5, 0.45, 0.6, 0.5)
    N = n[0] * n[1] * n[2]
    rng = np.random.default_rng(7)
    mu = 0.02 * rng.standard_normal((9, N))
    for d in (0, 4, 8):
        mu[d] -= 0.2
    mu, rhs = mu.reshape(-1), rng.standard_normal(3 * N)
    kw = dict(boundary_x=pg.BOUNDARY_WALL_OPEN) if wall else {}
    sim = pg.GpuSimulation(box, pg.IMPLICIT, particle_real=1, pressure_compat=0, tile=(0, 0, 0), **kw)
    x, info = sim.maxwell_solve(mu, rhs, pg.solve_opts(pg.GMRES_REFERENCE, max_iter=max_iter, tol=1e-8))
    again, _ = sim.maxwell_solve(mu, rhs, pg.solve_opts(pg.GMRES_REFERENCE, max_iter=max_iter, tol=1e-8))
    sim.close()
    assert np.array_equal(x, again)   # sums in a fixed order
    g = O.make_grid(box, pressure_compat=0, wall_x=1 if wall else 0)
    res = np.linalg.norm(O.maxwell_apply(g, mu, x) - rhs) / np.linalg.norm(rhs)
    assert abs(res - info["rel_residual"]) <= 1e-13
    assert info["iterations"] <= max_iter - 2
