"""FP64 explicit step of loads of which a few, many or all particles start on cell
faces: chunks that the fused kernel shares with its deferred pass, chunks left to that
whole, and mask words of every fill.  Needs a GB300."""
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


@pytest.mark.parametrize("n", [(8, 8, 8), (17, 9, 12), (24, 10, 1), (40, 32, 32)])
@pytest.mark.parametrize("share", [0.005, 0.1, 0.16, 0.22, 0.6, 1.0])
@pytest.mark.parametrize("cold", [False, True])
def test_loads_with_particles_on_faces_match_oracle(pg, n, share, cold):
    """`share` of the particles start on one, two or three faces (at rest there if
    cold); no fields, so that those have the oracle's velocities bit for bit.  The others
    start well inside their cells: there the fused kernel's roundings move the
    current by rounding only."""
    st = I.buneman_plasma(*n, ppc=5, seed=91)
    rng = np.random.default_rng(92)
    st.E = np.zeros_like(st.E)
    st.B = np.zeros_like(st.B)
    for sp in st.species:
        c = len(sp["ox"])
        on = rng.random(c) < share
        axes = rng.integers(1, 8, c)
        for a, k in enumerate(("ox", "oy", "oz")):
            sp[k] = np.where(on & (axes >> a & 1 == 1), 0.0, 0.05 + 0.9 * sp[k])
        if cold:
            for k in ("px", "py", "pz"):
                sp[k] = np.where(on, 0.0, sp[k])
    sim = pg.GpuSimulation(st.box, pg.BUNEMAN, particle_real=1, sort_every=1, tile=(0, 0, 0))
    sim.upload_state(st)
    sim.buneman_step(1)
    E, B, J = sim.download_fields()
    got = [sim.download_particles(s) for s in range(len(st.species))]
    sim.close()
    sp = copy_species(st.species)
    for s in sp:
        s["id"] = np.arange(len(s["cell"]), dtype=np.int32)
    Eo, Bo = st.E.copy(), st.B.copy()
    Jo = O.buneman_step(O.make_grid(st.box), sp, Eo, Bo)
    # rounding of sums of a few dozen terms; a particle on the other side moves J by
    # 1e-4 and more of the largest value, one left out or taken twice by as much
    assert rel_err(J, Jo.reshape(J.shape)) < 1e-12
    assert rel_err(E, Eo) < 1e-12
    for d, r in zip(got, sp):
        a, b = np.argsort(d["id"]), np.argsort(r["id"])
        for k, length in zip(range(3), (st.box.nx * st.box.dx, st.box.ny * st.box.dy, st.box.nz * st.box.dz)):
            far = np.abs(I.positions(st.box, d)[k][a] - I.positions(st.box, r)[k][b])
            assert np.minimum(far, length - far).max() < 1e-12 * length
