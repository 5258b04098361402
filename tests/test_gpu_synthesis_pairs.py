"""The profile kernel takes two models per warp; the two share a tile of the
PSF's product unless one is macroturbulent.  A model's profiles must not
depend on its partner or on its place: calls of an odd and an even number of
models, a model alone, and pairs of every mixture of v_mac on and off give the
same values, which are those of the response-function call and, to 1e-5 of
the Stokes-I norm, of the FP64 oracle -- one and two samples per lane, PSF and
stray light on and off, models in single and double precision."""
import numpy as np
import pytest

import gmilos_b200 as G
import helpers as H
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nl,psf,stray", [(30, True, True), (30, False, False), (8, True, False), (33, True, True),
                                          (64, False, True)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_profiles_do_not_depend_on_the_pair(nl, psf, stray, dtype):
    l0, zo = H.fe_line()
    lam, _ = H.grid(nl)
    p = O.psf_gauss(100.0, lam) if psf else None
    ocfg = O.make_cfg(lam, l0, zo, psf=p, init=H.GUESS)
    sl = H.stray_profile(ocfg) if stray else None
    n = 37
    t = H.truth_models(n, np.random.default_rng(nl), alpha_range=(0.7, 1.0) if stray else None)
    t[:, 9] = np.where(np.arange(n) % 5 < 2, 0.0, 0.9)   # pairs: off-off, on-on, on-off, off-on
    t = t.astype(dtype)
    with G.Engine(0) as e:
        e.configure(G.make_config(lam, l0, G.zeeman_from_levels(2, 1, 1.0, 2, 2, 0.0, 1.0), psf=p, init=H.GUESS,
                                  slight=sl))
        whole = e.synthesize(t)
        np.testing.assert_array_equal(e.synthesize(t[1:]), whole[1:])
        np.testing.assert_array_equal(e.synthesize(t[:1]), whole[:1])
        with_rf, rf = e.synthesize(t, rf=True)
        alone, rf_alone = e.synthesize(t[3:4], rf=True)
    np.testing.assert_array_equal(alone, with_rf[3:4])
    np.testing.assert_array_equal(rf_alone, rf[3:4])
    # the two kernels round differently: a few float roundings of the profile
    assert np.abs(with_rf - whole).max() < 1e-6
    for i in range(n):
        s64 = O.synth_d(ocfg, t[i].astype(np.float64), slight=None if sl is None else sl.astype(np.float64))
        assert H.rel_to_I(whole[i], s64).max() < 1e-5
