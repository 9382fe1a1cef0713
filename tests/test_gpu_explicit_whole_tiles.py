"""Fused explicit step of boxes with so many tiles that a CTA takes whole ones (more
than half as many as run at once: 304 with FP32 particles, 152 with FP64 ones), as
the large runs do; smaller boxes share tiles between CTAs.  Needs a GB300."""
import numpy as np
import pytest

import pyoracle as O
from fixtures import copy_species, rel_err, yee_physical
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


def away_from_faces(st, margin=0.02):
    """Particles that start or end a step within `margin` cells of a face rest in the
    middle of their cell along that axis: which side a rounding puts them on moves
    the current by far more than the rounding.  (Fields so weak that they move nothing
    by the margin.)"""
    b = st.box
    for sp in st.species:
        gam = np.sqrt(1 + (sp["px"] ** 2 + sp["py"] ** 2 + sp["pz"] ** 2) / sp["m"] ** 2)
        for o, p, d in (("ox", "px", b.dx), ("oy", "py", b.dy), ("oz", "pz", b.dz)):
            end = sp[o] + sp[p] / (sp["m"] * gam) * b.dt / d
            near = (np.minimum(sp[o], 1 - sp[o]) < margin) | (np.abs(end - np.round(end)) < margin)
            sp[o] = np.where(near, 0.5, sp[o]).astype(sp[o].dtype)
            sp[p] = np.where(near, 0.0, sp[p]).astype(sp[p].dtype)
    return st


def compare(sim, box, spo, E, B, J, real, wall):
    # FP64: sums of a few dozen terms after a handful of roundings each; FP32
    # particles and fields: 6e-8 each, the current's terms alternate in sign
    tol = 1e-11 if real else 1e-5
    Eg, Bg, Jg = sim.download_fields()
    pick = yee_physical if wall else lambda a, box, which: a
    assert rel_err(pick(Eg, box, "E"), pick(E, box, "E")) < tol
    assert rel_err(pick(Bg, box, "B"), pick(B, box, "B")) < tol
    assert rel_err(Jg, J.reshape(Jg.shape)) < tol
    for s, ref in enumerate(spo):
        got = sim.download_particles(s)
        a, b = np.argsort(got["id"]), np.argsort(ref["id"])
        assert np.array_equal(got["id"][a], ref["id"][b])
        for x, y, n, d in zip(I.positions(box, got), I.positions(box, ref), (box.nx, box.ny, box.nz), (box.dx, box.dy, box.dz)):
            far = np.abs(x[a] - y[b])
            assert np.minimum(far, n * d - far).max() < tol * n * d
        for k in ("px", "py", "pz"):
            assert rel_err(got[k][a], ref[k][b]) < tol


# 180 and 320 tiles of 8^3 with FP32 particles (whole tiles, one wave and two), 100
# with FP64 ones; tiles of another shape by name (run-time extents)
@pytest.mark.parametrize("n,real,tile", [((48, 48, 40), 0, (0, 0, 0)), ((64, 40, 64), 0, (0, 0, 0)),
                                         ((40, 40, 32), 1, (0, 0, 0)), ((32, 40, 32), 0, (8, 8, 4)),
                                         ((32, 24, 32), 1, (8, 8, 4))])
def test_periodic_box_matches_oracle(pg, n, real, tile):
    st = I.buneman_plasma(*n, ppc=1, sigma=1e-3, seed=81)
    rng = np.random.default_rng(82)
    st.E = st.E + 0.02 * rng.standard_normal(st.E.shape)
    st.B = st.B + 0.02 * rng.standard_normal(st.B.shape)
    away_from_faces(st)
    sim = pg.GpuSimulation(st.box, pg.BUNEMAN, particle_real=real, sort_every=1, tile=tile)
    sim.upload_state(st)
    sim.buneman_step(1)
    spo = copy_species(st.species)
    for sp in spo:
        sp["id"] = np.arange(len(sp["cell"]), dtype=np.int32)
    E, B = st.E.copy(), st.B.copy()
    J = O.buneman_step(O.make_grid(st.box), spo, E, B)
    compare(sim, st.box, spo, E, B, J, real, False)
    sim.close()


# 162 tiles with FP32 particles, 112 with FP64 ones
@pytest.mark.parametrize("n,real", [((72, 48, 24), 0), ((56, 32, 32), 1)])
def test_wall_box_matches_oracle(pg, n, real):
    st = away_from_faces(I.shock_plasma(*n, dx=0.5, dt=0.225, ppc=(1, 1, 1), flow_gamma=3.0, theta_e=0.3, sigma=1e-3, seed=83,
                                        first_cell=I.TRISTAN_WALL_NODE))
    sim = pg.GpuSimulation(st.box, pg.BUNEMAN, particle_real=real, sort_every=1, tile=(0, 0, 0),
                           boundary_x=pg.BOUNDARY_WALL_OPEN, e_right=st.e_right, b_right=st.b_right)
    sim.upload_state(st)
    sim.buneman_step(1)
    spo = copy_species(st.species)
    for sp in spo:
        sp["id"] = np.arange(len(sp["cell"]), dtype=np.int32)
    E, B = st.E.copy(), st.B.copy()
    J = O.buneman_step(O.make_grid(st.box, wall_x=1, e_right=st.e_right, b_right=st.b_right), spo, E, B)
    compare(sim, st.box, spo, E, B, J, real, True)
    sim.close()
