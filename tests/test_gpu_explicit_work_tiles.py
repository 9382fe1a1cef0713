"""The fused explicit kernel in work tiles of 8^3 cells, which a box takes by its number of
tiles and particles (csrc/explicit_split.hpp): against the oracle and against the same
tiles of the sort asked for by name, on both sides of the rule.  Needs a GB300."""
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


def divisor(n):
    return next(t for t in (8, 4, 2, 1) if n % t == 0)


def state(n, ppc, seed=61):
    st = I.buneman_plasma(*n, ppc=ppc, sigma=1e-3, seed=seed)
    rng = np.random.default_rng(seed + 1)
    st.E = st.E + 0.05 * rng.standard_normal(st.E.shape)
    st.B = st.B + 0.05 * rng.standard_normal(st.B.shape)
    # cells of every fill: the particles of half the cells moved to the next one
    for sp in st.species:
        sp["cell"] = np.where(sp["cell"] % 2 == 0, sp["cell"], sp["cell"] - 1).astype(sp["cell"].dtype)
    return st


def run(pg, st, real, tile, steps, every=1):
    sim = pg.GpuSimulation(st.box, pg.BUNEMAN, particle_real=real, sort_every=every, tile=tile)
    sim.upload_state(st)
    sim.buneman_step(steps)
    out = sim.download_fields()
    sim.close()
    return out


# more than 3,000 tiles: always in work tiles, ragged by 1 to 7 cells, an axis of one work
# tile and a cell among them; 26^3 and 44x20x44 with few particles: by the estimate
@pytest.mark.parametrize("n,ppc", [((15, 15, 15), 5), ((9, 17, 33), 4), ((11, 13, 23), 3), ((60, 15, 9), 2), ((26, 26, 26), 1),
                                   ((44, 60, 44), 1)])
@pytest.mark.parametrize("real", [0, 1])
def test_work_tiles_give_what_the_sorts_tiles_give(pg, n, ppc, real):
    st = state(n, ppc)
    got = run(pg, st, real, (0, 0, 0), 3)
    ref = run(pg, st, real, tuple(divisor(a) for a in n), 3)
    for a, b in zip(got, ref):
        if real == 0:   # integer sums of the same runs, nothing deferred
            assert np.array_equal(a, b)
        else:           # sums in another order: 1e-16 each over at most a few hundred terms
            assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


@pytest.mark.parametrize("n,ppc", [((15, 15, 15), 5), ((9, 17, 33), 4), ((26, 26, 26), 1), ((26, 26, 26), 24), ((20, 12, 28), 6)])
def test_either_choice_matches_oracle(pg, n, ppc):
    """One FP64 step; 26^3 takes work tiles with one particle per species and cell, the
    sort's tiles with 24."""
    st = state(n, ppc)
    E, B, J = run(pg, st, 1, (0, 0, 0), 1)
    Eo, Bo = st.E.copy(), st.B.copy()
    Jo = O.buneman_step(O.make_grid(st.box), copy_species(st.species), Eo, Bo)
    # a few dozen terms per sum, a handful of roundings each
    assert rel_err(J, Jo.reshape(J.shape)) < 1e-11
    assert rel_err(E, Eo) < 1e-11
    assert rel_err(B, Bo) < 1e-11
