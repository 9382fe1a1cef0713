"""The fused explicit kernel's work tiles of 8^3 cells, taken where an axis is no
multiple of 8 and the caller left the tiles to the library, against one CTA per
tile of the sort (the same tiles asked for by name).  Needs a GB300."""
import numpy as np
import pytest

from picpp_gb300 import initstate as I

pytestmark = pytest.mark.gpu

# extents from one cell past a work tile to one cell short of two, mixed with
# whole ones; tiles of the sort of 1, 2, 4 and 8 cells
BOXES = [(9, 9, 9), (8, 15, 10), (20, 8, 9), (36, 12, 14), (16, 8, 60)]


@pytest.fixture(scope="module")
def pg():
    import picpp_gb300 as P
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    P.load_library()
    return P


def divisor(n):
    return next(t for t in (8, 4, 2, 1) if n % t == 0)


def run(pg, st, real, tile, every, steps):
    sim = pg.GpuSimulation(st.box, pg.BUNEMAN, particle_real=real, sort_every=every, tile=tile)
    sim.upload_state(st)
    sim.buneman_step(steps)
    out = sim.download_fields()
    parts = []
    for s in range(len(st.species)):
        p = sim.download_particles(s)
        o = np.argsort(p["id"])
        parts.append({k: v[o] for k, v in p.items()})
    sim.close()
    return out, parts


@pytest.mark.parametrize("n", BOXES)
@pytest.mark.parametrize("real", [0, 1])
@pytest.mark.parametrize("every,px", [(1, 0.0), (4, 5.0)])
def test_work_tiles_match_one_cta_per_tile(pg, n, real, every, px):
    """px = 5 m c beams sorted every fourth step: particles leave their tiles and
    take the deferred pass, whose sums (FP64 atomics) come in any order."""
    st = I.buneman_plasma(*n, ppc=5, seed=51)
    rng = np.random.default_rng(9)
    st.E = st.E + 0.05 * rng.standard_normal(st.E.shape)
    st.B = st.B + 0.05 * rng.standard_normal(st.B.shape)
    # cells of every fill: the particles of half the cells moved to the next one
    for sp in st.species:
        sp["cell"] = np.where(sp["cell"] % 2 == 0, sp["cell"], sp["cell"] - 1).astype(sp["cell"].dtype)
        if px:
            sp["px"] = np.where(np.arange(len(sp["px"])) % 2 == 0, 1.0, -1.0) * px * sp["m"] + 0.1 * sp["px"]
    tile = tuple(divisor(a) for a in n)
    got, gp = run(pg, st, real, (0, 0, 0), every, 3)
    ref, rp = run(pg, st, real, tile, every, 3)
    if real == 0 and not px:   # integer sums of the same runs, nothing deferred
        for a, b in zip(got, ref):
            assert np.array_equal(a, b)
        for a, b in zip(gp, rp):
            for k in a:
                assert np.array_equal(a[k], b[k]), k
    else:
        # FP64: sums in another order, 1e-16 each over at most a few hundred
        # terms.  FP32 with deferred particles: such a difference may round an
        # FP32 field value or a position the other way (6e-8), and three steps
        # of it stay below 1e-5 of the largest value.
        tol = 1e-12 if real else 1e-5
        for a, b in zip(got, ref):
            assert np.abs(a - b).max() <= tol * np.abs(b).max()
