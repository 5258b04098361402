"""The 11-term solve where the elimination gives way to the Jacobi solve
(a pivot below 1e-10 of its diagonal, negative or not a number): one LM step
from start models that are not numbers, and undamped steps whose normal
matrices are singular to FP32, among ordinary pixels.  A pixel's step must not
depend on its place or its neighbours, bit for bit."""
import numpy as np
import pytest

import gmilos_b200 as G
import helpers as H
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nl", [30, 45])
@pytest.mark.parametrize("flambda", [0.1, 1e-13])
def test_steps_do_not_depend_on_the_neighbours(nl, flambda):
    rng = np.random.default_rng(nl)
    l0, zo = H.fe_line()
    lam, _ = H.grid(nl)
    psf = O.psf_gauss(100.0, lam)
    init = H.GUESS[:9] + (0.6, 1.0)
    fix = (1,) * 11
    ocfg = O.make_cfg(lam, l0, zo, psf=psf, fix=fix, init=init)
    sl = H.stray_profile(ocfg)
    n = 515
    t = H.truth_models(n, rng, alpha_range=(0.7, 1.0))
    t[:, 9] = rng.uniform(0.2, 3.0, n)
    obs = H.observations(ocfg, t, rng, slight=sl)
    start = t * rng.uniform(0.98, 1.02, t.shape)
    start[::5, 1] = 0.0          # no polarisation: the angles' rows are zero
    bad = np.arange(n) % 7 == 3
    start[bad, 4] = np.nan
    with G.Engine(0) as e:
        e.configure(G.make_config(lam, l0, G.zeeman_from_levels(2, 1, 1.0, 2, 2, 0.0, 1.0), psf=psf, fix=fix,
                                  init=init, slight=sl))
        whole = e.lm_step(obs, start, flambda)
        order = rng.permutation(n)
        moved = e.lm_step(obs[order], start[order], flambda)
        clean = e.lm_step(obs[~bad], start[~bad], flambda)
    for a, b, c in zip(whole, moved, clean):
        np.testing.assert_array_equal(b, a[order])
        np.testing.assert_array_equal(c, a[~bad])
    assert np.isfinite(whole[0][~bad]).all() and np.isnan(whole[0][bad]).any(axis=1).all()
