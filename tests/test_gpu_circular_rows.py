"""The circular convolution of macroturbulence, five outputs a lane: profiles
and response functions at the grid lengths where its last group of outputs,
its last taps or its last batch of rows are partial, one and two samples per
lane, with the PSF folded into the kernel and without, against the FP64
oracle: synthesis <= 1e-5 of the Stokes-I norm and response functions <=
max(1e-4, 10 x the FP32 oracle's own deviation), the bars of the other
macroturbulence tests."""
import numpy as np
import pytest

import gmilos_b200 as G
import helpers as H
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nl", [5, 9, 11, 29, 32, 33, 36, 63, 64])
@pytest.mark.parametrize("psf", [False, True])
def test_profiles_and_response_functions_at_grid_edges(nl, psf):
    l0, zo = H.fe_line()
    lam, _ = H.grid(nl)
    p = O.psf_gauss(100.0, lam) if psf else None
    init = list(H.GUESS)
    init[9] = 0.6
    fix = (1,) * 11
    ocfg = O.make_cfg(lam, l0, zo, psf=p, fix=fix, init=init)
    t = H.truth_models(24, np.random.default_rng(nl))
    t[:, 9] = np.linspace(0.3, 3.0, len(t))
    with G.Engine(0) as e:
        e.configure(G.make_config(lam, l0, G.zeeman_from_levels(2, 1, 1.0, 2, 2, 0.0, 1.0), psf=p, fix=fix, init=init))
        s, rf = e.synthesize(t, rf=True)
    for i, m in enumerate(t):
        s64, r64 = O.synth_d(ocfg, m, rf=True)
        _, r32 = O.synth_f(ocfg, m, rf=True)
        assert H.rel_to_I(s[i], s64).max() < 1e-5
        own = H.rf_rel(r32, r64)
        assert (H.rf_rel(rf[i], r64) <= np.maximum(1e-4, 10 * own)).all()
