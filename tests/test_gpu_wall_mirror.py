"""A wall box whose field throws a particle so far that its mirror image lies
beyond the open boundary: the particle has escaped.  Needs a GB300."""
import numpy as np
import pytest

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


@pytest.mark.parametrize("real", [0, 1])
@pytest.mark.parametrize("sort_every", [0, 1])
@pytest.mark.parametrize("ex", [-1e3, -1e5, -1e12])
def test_particles_mirrored_beyond_the_open_boundary_escape(pg, real, sort_every, ex):
    """Particles at rest in a field E_x: with next to no charge on the grid E
    stays what it is, and the Picard velocity q dt E / 2 m = |ex| / 5 puts the
    mirror image about 0.08 |ex| cells right of the wall, beyond the 12 physical
    ones.  The predictor moves less than a cell and so reflects none of cells 2 up."""
    n = (14, 6, 4)
    box = I.Box(*n, 0.5, 0.5, 0.5, 0.4, theta=0.5)
    sim = pg.GpuSimulation(box, pg.IMPLICIT, particle_real=real, pressure_compat=0, sort_every=sort_every, tile=(0, 0, 0),
                           boundary_x=pg.BOUNDARY_WALL_OPEN, e_right=(ex, 0.0, 0.0), b_right=(0.0, 0.0, 0.0))
    cells = np.arange(box.ncells)
    cells = cells[(cells % n[0] >= 2) & (cells % n[0] < n[0] - 4)].astype(np.int32)
    rng = np.random.default_rng(3)
    off = [rng.random(len(cells)) for _ in range(3)]
    sp = dict(cell=cells, ox=off[0], oy=off[1], oz=off[2], px=np.zeros(len(cells)), py=np.zeros(len(cells)),
              pz=np.zeros(len(cells)))
    sim.add_species(1.0, 1.0, 1e-30, len(cells))
    sim.upload_particles(0, sp)
    E = np.zeros((3, n[2], n[1], n[0]))
    E[0] = ex
    sim.upload_fields(E, np.zeros_like(E))
    for _ in range(2):   # the second step sorts what the first left
        sim.implicit_step(pg.solve_opts(pg.GMRES_RESTARTED))
    assert len(sim.download_particles(0)["cell"]) == 0
    sim.close()
