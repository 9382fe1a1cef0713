"""FP64 explicit step of particles that start exactly on cell faces: the zigzag
split of the fused kernel and its deferred pass falls on the oracle's side of
the face.  Needs a GB300."""
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


@pytest.mark.parametrize("n,tile", [((8, 8, 8), (0, 0, 0)), ((17, 9, 12), (0, 0, 0)), ((12, 8, 8), (4, 4, 4)),
                                    ((16, 12, 1), (0, 0, 0))])
def test_particles_on_faces_match_oracle(pg, n, tile):
    """Offsets in quarters, a quarter of them 0 along each axis; no fields, so that
    the velocities are the oracle's bit for bit and the current is what is compared."""
    st = I.buneman_plasma(*n, ppc=6, seed=71)
    rng = np.random.default_rng(72)
    st.E = np.zeros_like(st.E)
    st.B = np.zeros_like(st.B)
    for sp in st.species:
        for k in ("ox", "oy", "oz"):
            sp[k] = rng.integers(0, 4, len(sp[k])) / 4.0
    sim = pg.GpuSimulation(st.box, pg.BUNEMAN, particle_real=1, sort_every=1, tile=tile)
    sim.upload_state(st)
    sim.buneman_step(1)
    E, B, J = sim.download_fields()
    sim.close()
    sp = copy_species(st.species)
    Eo, Bo = st.E.copy(), st.B.copy()
    Jo = O.buneman_step(O.make_grid(st.box), sp, Eo, Bo)
    # rounding of sums of a few dozen terms; a particle on the other side moves J by
    # 1e-4 and more of the largest value
    assert rel_err(J, Jo.reshape(J.shape)) < 1e-12
    assert rel_err(E, Eo) < 1e-12
