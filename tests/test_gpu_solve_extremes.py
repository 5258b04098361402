"""The solve kernel (one thread per system, step limits by that thread) against
the solve in the trial kernel (half-warps, limits by a warp) where data are not
profiles: noise far above the signal, so that steps run into every limit and
range check; observations that are not numbers or infinite; flat zero
profiles; one free parameter; damping that follows chi2 (logclambda).  A call
just below 24 576 pixels and one above it must give the same results bit for
bit, both 10-term variants, one and two samples per lane."""
import numpy as np
import pytest

import gmilos_b200 as G
import helpers as H
import oracle as O

pytestmark = pytest.mark.gpu

ZG = G.zeeman_from_levels(2, 1, 1.0, 2, 2, 0.0, 1.0)
KEYS = ("model64", "chi2", "iters", "accepted", "status")
EDGE = 24575
ONE = (0, 1) + (0,) * 9
TEN = (1,) * 9 + (0, 1)


@pytest.mark.parametrize("nl,fix,vmac,kw", [
    (30, H.FREE9, 0.0, {}), (30, TEN, 0.0, dict(numerics=1)), (30, TEN, 0.8, dict(logclambda=1)), (30, ONE, 0.0, {}),
    (30, (0,) * 11, 0.0, {}), (45, H.FREE9, 0.0, dict(logclambda=1)), (45, TEN, 0.8, {})])
def test_either_side_of_the_edge_agrees(nl, fix, vmac, kw):
    rng = np.random.default_rng(nl + sum(fix))
    l0, zo = H.fe_line()
    lam, _ = H.grid(nl)
    psf = O.psf_gauss(100.0, lam)
    init = H.GUESS[:9] + (vmac, 1.0)
    n = 701
    t = H.truth_models(n, rng)
    obs = H.observations(O.make_cfg(lam, l0, zo, psf=psf, init=init), t, rng)
    scale = 10.0 ** rng.uniform(-2, 3, (n, 1, 1))
    obs = (obs + scale * rng.normal(0, 1, obs.shape)).astype(np.float32)
    obs[5], obs[17, 2, 3], obs[31, 0], obs[47] = np.nan, np.inf, -np.inf, 0.0
    idx = np.arange(EDGE + 18) % n
    cube = np.ascontiguousarray(obs[idx])
    sl = H.stray_profile(O.make_cfg(lam, l0, zo, psf=psf, init=init)) if fix[10] else None
    with G.Engine(0) as e:
        e.configure(G.make_config(lam, l0, ZG, psf=psf, init=init, fix=fix, slight=sl, miter=14, **kw))
        small = e.invert(cube[:EDGE])
        two = e.stats()["kernel_launches"] // 14
        large = e.invert(cube)
        assert two == 2 and e.stats()["kernel_launches"] // 14 == 3
    for k in KEYS:
        np.testing.assert_array_equal(large[k][:EDGE], small[k], err_msg=k)
        np.testing.assert_array_equal(large[k], large[k][:n][idx], err_msg=k)
    m = large["model64"][:n]
    if sum(fix) > 1:   # limits and range checks were met
        assert (m[:, 0] == 1).any() and (np.abs(m[:, 2]) == 20).any() and (m[:, 8] == 2.0).any()
