"""Response functions under stray light carry the filling factor as it is, a
double: those of a model with factor a are the ones with factor 1, times a in
double, rounded once -- for ordinary factors and for ones beyond the range of
a float, at 10 and 11 terms, one and two samples per lane."""
import numpy as np
import pytest

import gmilos_b200 as G
import helpers as H
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nl,eleven", [(30, False), (30, True), (45, False)])
def test_the_filling_factor_scales_in_double(nl, eleven):
    rng = np.random.default_rng(nl)
    l0, zo = H.fe_line()
    lam, _ = H.grid(nl)
    psf = O.psf_gauss(100.0, lam)
    sl = H.stray_profile(O.make_cfg(lam, l0, zo, psf=psf, init=H.GUESS))
    n = 3000
    t = H.truth_models(n, rng, alpha_range=(0.0, 1.0))
    t[:10, 10] = (0.0, 1e-12, 1e-50, 1e30, 3.5e38, 1e39, -1e39, 1e300, np.inf, np.nan)
    one = t.copy()
    one[:, 10] = 1.0
    with G.Engine(0) as e:
        e.configure(G.make_config(lam, l0, G.zeeman_from_levels(2, 1, 1.0, 2, 2, 0.0, 1.0), psf=psf, init=H.GUESS,
                                  slight=sl, fix=(1,) * 11 if eleven else H.FREE9))
        _, got = e.synthesize(t, rf=True)
        _, base = e.synthesize(one, rf=True)
    terms = list(range(10 if eleven else 9))
    with np.errstate(all="ignore"):
        want = (base[:, :, terms].astype(np.float64) * t[:, 10, None, None, None]).astype(np.float32)
    got = got[:, :, terms]
    tiny = np.abs(want) < 1.2e-38          # the engine flushes these to zero
    np.testing.assert_array_equal(got[~tiny], want[~tiny])
    assert (np.abs(got[tiny]) < 1.2e-38).all()
