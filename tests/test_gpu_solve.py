"""The solve kernel of the wave-synchronous inversion: one thread per 10x10
system, 16 pixels with two dampings each to a warp, for chunks of 24 576
pixels and more.  It repeats the operations of the half-warp solve in the trial
kernel, which smaller chunks run, in the same order: a call of 16 384 pixels
and calls of a few more must give the same results for the first 16 384 bit
for bit, for every free mask, both numerics modes, both 10-term variants, one
and two samples per lane, and however full the last warp is."""
import numpy as np
import pytest

import gmilos_b200 as G
import helpers as H
import oracle as O

pytestmark = pytest.mark.gpu

ZG = G.zeeman_from_levels(2, 1, 1.0, 2, 2, 0.0, 1.0)
KEYS = ("model64", "chi2", "iters", "accepted", "status")
EDGE = 24575
MASKS = {"nine": H.FREE9, "seven": (1, 1, 1, 1, 1, 1, 1, 0, 0, 0, 1), "field": (0, 1, 0, 0, 0, 1, 1, 0, 0, 0, 0),
         "angles fixed": (1, 1, 1, 1, 1, 0, 0, 1, 1, 0, 1)}


@pytest.fixture(scope="module")
def engine():
    e = G.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("nl,numerics,mask,given,more", [
    (30, 0, "nine", False, 1), (30, 0, "seven", True, 15), (30, 0, "field", False, 16), (30, 1, "nine", True, 17),
    (30, 1, "angles fixed", False, 33), (45, 0, "nine", False, 49), (45, 1, "seven", True, 31)])
def test_chunks_on_either_side_of_the_edge_agree(engine, nl, numerics, mask, given, more):
    lam, _ = H.grid(nl)
    l0, zo = H.fe_line()
    psf = O.psf_gauss(100.0, lam)
    rng = np.random.default_rng(17)
    some = H.truth_models(701, rng)
    obs = H.observations(O.make_cfg(lam, l0, zo, psf=psf, init=H.GUESS), some, rng)
    idx = np.arange(EDGE + more) % len(some)
    cube = np.ascontiguousarray(obs[idx])
    start = np.ascontiguousarray(some[idx] * 1.02 + 0.01) if given else None
    engine.configure(G.make_config(lam, l0, ZG, psf=psf, init=H.GUESS, fix=MASKS[mask], numerics=numerics, miter=14))
    small = engine.invert(cube[:EDGE], init_models=None if start is None else start[:EDGE])
    per_wave = engine.stats()["kernel_launches"] // 14
    large = engine.invert(cube, init_models=start)
    assert per_wave == 2 and engine.stats()["kernel_launches"] // 14 == 3
    for k in KEYS:
        np.testing.assert_array_equal(large[k][:EDGE], small[k], err_msg=k)
        # the same pixel at another place of the list
        np.testing.assert_array_equal(large[k], large[k][:len(some)][idx], err_msg=k)
