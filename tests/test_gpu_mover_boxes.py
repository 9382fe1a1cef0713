"""The implicit mover's work boxes (csrc/implicit_tile.cuh) on grids whose axes 8
does not divide, against one CTA per tile of the sort (the same tiles asked for
by name); and a two-cell periodic axis, whose halo wraps around it more than
once, against the oracle.  Needs a GB300."""
import numpy as np
import pytest

import pyoracle as O
from picpp_gb300 import initstate as I
from fixtures import copy_species, periodic_dist, rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pg():
    import picpp_gb300 as P
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    P.load_library()
    return P


def state(n, ppc, dt=0.4, gamma=4.0):
    st = I.beams_plasma(*n, ppc=ppc, beam_gamma=gamma, dt=dt, seed=61)
    rng = np.random.default_rng(62)
    st.E = st.E + 0.05 * rng.standard_normal(st.E.shape)
    st.B = st.B + 0.05 * rng.standard_normal(st.B.shape)
    for sp in st.species:   # all directions, so that particles leave their tiles along every axis
        sp["py"] = sp["py"] + sp["m"] * rng.standard_normal(len(sp["py"]))
        sp["pz"] = sp["pz"] + sp["m"] * rng.standard_normal(len(sp["pz"]))
    return st


def by_id(d):
    o = np.argsort(d["id"])
    return {k: v[o] for k, v in d.items()}


def distances(box, a, b):
    for x, y, l, d in zip(I.positions(box, a), I.positions(box, b), (box.nx, box.ny, box.nz), (box.dx, box.dy, box.dz)):
        yield periodic_dist(x, y, l * d).max() / d


def divisor(n):
    return next(t for t in (8, 4, 2, 1) if n % t == 0)


@pytest.mark.parametrize("n,ppc", [((9, 9, 9), 3), ((20, 7, 3), 9), ((36, 12, 10), 2), ((33, 15, 1), 40), ((3, 5, 17), 33)])
@pytest.mark.parametrize("real", [0, 1])
@pytest.mark.parametrize("every", [1, 3])
def test_work_boxes_match_one_cta_per_tile(pg, n, ppc, real, every):
    st = state(n, ppc)
    out = []
    for tile in ((0, 0, 0), tuple(divisor(a) for a in n)):
        sim = pg.GpuSimulation(st.box, pg.IMPLICIT, particle_real=real, pressure_compat=0, sort_every=every, tile=tile)
        sim.upload_state(st)
        for _ in range(3):
            sim.implicit_step(pg.solve_opts(pg.GMRES_RESTARTED, tol=1e-13))
        out.append([by_id(sim.download_particles(s)) for s in range(2)])
        sim.close()
    # the movers do the same arithmetic; the moments' sums come in another order
    # (FP64 1e-16 a term, FP32 6e-8), which the solve passes on at its condition
    # number (about 10) in each of three steps
    tol = 1e-11 if real else 1e-5
    for a, b in zip(*out):
        assert max(distances(st.box, a, b)) <= tol
        for k in ("px", "py", "pz"):
            assert rel_err(a[k], b[k]) <= tol


@pytest.mark.parametrize("n", [(9, 2, 2), (2, 9, 1), (8, 2, 3)])
def test_two_cell_axes_match_oracle(pg, n):
    """dt = 3.2 dx / c: trial positions up to 1.6 cells away."""
    st = state(n, 9, dt=1.6)
    sim = pg.GpuSimulation(st.box, pg.IMPLICIT, particle_real=1, pressure_compat=0, sort_every=1, tile=(0, 0, 0))
    sim.upload_state(st)
    sim.implicit_step(pg.solve_opts(pg.GMRES_REFERENCE))
    g = O.make_grid(st.box, pressure_compat=0)
    sp = copy_species(st.species)
    E, B = st.E.reshape(-1).copy(), st.B.reshape(-1).copy()
    O.implicit_step(g, sp, E, B)
    Eg, Bg, _ = sim.download_fields()
    # the solves stop at the same residual (1e-8 / dim, at least 1e-15); the rest is
    # rounding, as in every other step against the oracle
    assert rel_err(Eg.reshape(-1), E) < 1e-11
    for s in range(2):
        got = by_id(sim.download_particles(s))
        assert max(distances(st.box, got, sp[s])) < 1e-11
        for k in ("px", "py", "pz"):
            assert rel_err(got[k], sp[s][k]) < 1e-11
    sim.close()
