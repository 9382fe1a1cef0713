"""Density, energy and velocity moments of small boxes with many particles per cell, where
the deposit's warps begin at different corners, on both sides of that rule.  Needs a
GB300."""
import numpy as np
import pytest

import pyoracle as O
from fixtures import copy_species, rel_err
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


@pytest.mark.parametrize("n,ppc", [((8, 8, 8), 19), ((8, 8, 8), 20), ((5, 3, 7), 260), ((9, 6, 1), 150), ((40, 1, 1), 333),
                                   ((16, 16, 16), 30), ((16, 16, 17), 30)])
@pytest.mark.parametrize("real", [0, 1])
def test_moments_match_oracle(pg, n, ppc, real):
    st = I.buneman_plasma(*n, ppc=ppc, seed=31)
    for sp in st.species:   # values that FP32 particles hold too
        for k in ("ox", "oy", "oz", "px", "py", "pz"):
            sp[k] = sp[k].astype(np.float32).astype(np.float64)
            if k[0] == "o":
                sp[k] = np.minimum(sp[k], 1 - 2.0 ** -24)
    sim = pg.GpuSimulation(st.box, pg.BUNEMAN, particle_real=real, tile=(0, 0, 0))
    sim.upload_state(st)
    sim.updateDensityParameters()
    conc, en, vel, rho = O.density_moments(O.make_grid(st.box), copy_species(st.species))
    # FP64 sums of some thousand terms of either precision's weights: FP32 weights round
    # to 6e-8 each; the velocities' terms nearly cancel
    tol = 1e-11 if real else 1e-5
    for s in range(len(st.species)):
        c, e, v, r = sim.download_density(s)
        assert rel_err(c, conc[s]) < tol
        assert rel_err(e, en[s]) < tol
        assert np.abs(v - vel[s].reshape(v.shape)).max() < tol * max(np.abs(vel[s]).max(), 1.0)
    # (one species' charge density is 1 / 4 pi; the sum of both nearly cancels)
    assert np.abs(r - rho.reshape(r.shape)).max() < tol * max(np.abs(rho).max(), 1 / (4 * np.pi))
    sim.close()
