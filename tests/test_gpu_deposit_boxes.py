"""Boxes of cells of the staged implicit deposit (csrc/api.cu, deposit_boxes):
grids whose axes leave ragged boxes, boxes cut to single cells and boxes that
span a whole periodic axis, against the oracle.  Needs a GB300."""
import numpy as np
import pytest

import pyoracle as O
from picpp_gb300 import initstate as I
from fixtures import copy_species, rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pg():
    import picpp_gb300 as P
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    P.load_library()
    return P


@pytest.mark.parametrize("n,ppc", [((3, 1, 1), 40), ((17, 9, 1), 9), ((2, 2, 2), 70), ((9, 9, 9), 5), ((26, 5, 3), 33),
                                   ((33, 31, 4), 3), ((16, 24, 40), 2), ((41, 23, 18), 3)])
@pytest.mark.parametrize("real", [0, 1])
@pytest.mark.parametrize("wall", [False, True])
def test_staged_moments_match_oracle(pg, n, ppc, real, wall):
    if wall and min(n[0] - 3, n[1] - 1, n[2] - 1) < 1:
        pytest.skip("a wall box has three axes")
    st = I.beams_plasma(*n, ppc=ppc, beam_gamma=2.0, dt=0.2, seed=43)
    rng = np.random.default_rng(44)
    st.E = st.E + 0.05 * rng.standard_normal(st.E.shape)
    st.B = st.B + 0.05 * rng.standard_normal(st.B.shape)
    kw = dict(boundary_x=pg.BOUNDARY_WALL_OPEN) if wall else {}
    if wall:   # the two ghost columns are empty
        for sp in st.species:
            i = sp["cell"] % n[0]
            sp["cell"] = np.where(i >= n[0] - 2, sp["cell"] - 2, sp["cell"]).astype(np.int32)
    sim = pg.GpuSimulation(st.box, pg.IMPLICIT, particle_real=real, pressure_compat=0, sort_every=1, tile=(0, 0, 0), **kw)
    sim.upload_state(st)
    sim.updateElectroMagneticParameters()
    J, mu, rho, rhs = sim.download_moments()
    sim.close()
    g = O.make_grid(st.box, pressure_compat=0, wall_x=1 if wall else 0)
    E, B = st.E.reshape(-1).copy(), st.B.reshape(-1).copy()
    Jo, muo, rhoo, Pio, raw = O.implicit_moments(g, copy_species(st.species), E, B)
    # sums of a few hundred FP64 terms; FP32 particles, fields and run sums: 6e-8
    # a term, amplified by the cancellation of the beams' opposite currents
    tol = 1e-12 if real else 1e-5
    assert rel_err(mu, muo) < tol
    assert rel_err(J, Jo) < tol
    # (rho: each species' charge density is 1 / 4 pi; in a neutral box their sum
    # cancels to less than what FP32 accumulators resolve to 1e-5)
    assert np.abs(rho - rhoo).max() < tol * max(np.abs(rhoo).max(), 1 / (4 * np.pi))
