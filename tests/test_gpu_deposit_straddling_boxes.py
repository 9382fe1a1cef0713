"""Staged FP32 deposit in boxes that straddle the caller's tiles: the sums of a
cell's particles meet in FP64, so the moments do not depend on the tiles beyond FP64
rounding.  Needs a GB300."""
import numpy as np
import pytest

from picpp_gb300 import initstate as I
from fixtures import rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pg():
    import picpp_gb300 as P
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    P.load_library()
    return P


def moments(pg, st, tile):
    sim = pg.GpuSimulation(st.box, pg.IMPLICIT, particle_real=0, pressure_compat=0, sort_every=1, tile=tile)
    sim.upload_state(st)
    sim.updateElectroMagneticParameters()
    out = sim.download_moments()
    sim.close()
    return out


def test_moments_of_straddling_boxes_are_those_of_single_cells(pg):
    """15^3 cells in tiles of 5^3 are cut into boxes of 3^3, in tiles of one cell into boxes
    of several tiles: the same FP32 sums per cell and species, in the order of the
    particles' numbers, met in FP64 accumulators by either."""
    st = I.beams_plasma(15, 15, 15, ppc=11, beam_gamma=2.0, dt=0.2, seed=43)
    rng = np.random.default_rng(44)
    st.E = st.E + 0.05 * rng.standard_normal(st.E.shape)
    st.B = st.B + 0.05 * rng.standard_normal(st.B.shape)
    a, b = moments(pg, st, (5, 5, 5)), moments(pg, st, (1, 1, 1))
    # a few dozen FP64 additions of either sign per entry: 1e-16 each; FP32
    # accumulators differ by 1e-8 and more
    for x, y in zip(a, b):
        assert rel_err(x, y) < 1e-12
