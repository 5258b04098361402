"""Profiles of few models, one to a warp, and of more, two to a warp: at the
last count of the one and the first two of the other, every model's profiles
are the same bit for bit -- pairs of every mixture of v_mac on and off, an odd
and an even count, PSF on and off, one stray-light profile or a map, one
wavelength grid or one per model, models in single and double precision."""
import numpy as np
import pytest

import gmilos_b200 as G
import helpers as H
import oracle as O

pytestmark = pytest.mark.gpu

ZG = G.zeeman_from_levels(2, 1, 1.0, 2, 2, 0.0, 1.0)


@pytest.mark.parametrize("nl,psf,stray,grids,dtype", [
    (30, True, "profile", False, np.float64), (30, True, "map", True, np.float64), (30, False, "map", False, np.float32),
    (12, True, None, True, np.float32), (45, True, "map", True, np.float64), (64, False, None, False, np.float64),
    (49, True, "profile", False, np.float32)])
def test_either_side_of_the_edge_agrees(nl, psf, stray, grids, dtype):
    torch = pytest.importorskip("torch")
    edge = (16 if nl <= 32 else 12) * torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(nl)
    l0, zo = H.fe_line()
    lam, _ = H.grid(nl)
    p = O.psf_gauss(100.0, lam) if psf else None
    n = 37
    t = H.truth_models(n, rng, alpha_range=(0.7, 1.0) if stray else None)
    t[:, 9] = np.where(np.arange(n) % 5 < 2, 0.0, 0.9)   # pairs: off-off, on-on, on-off, off-on
    t = t.astype(dtype)
    one = H.stray_profile(O.make_cfg(lam, l0, zo, psf=p, init=H.GUESS))
    maps = (one * rng.uniform(0.9, 1.1, (n, 1, 1))).astype(np.float32)
    own = lam + rng.uniform(-0.02, 0.02, (n, 1))

    def profiles(e, idx):
        kw = {}
        if stray:
            kw = dict(slight=maps[idx] if stray == "map" else one, slight_per_pixel=stray == "map")
        if grids:
            kw["lambda_map"] = np.ascontiguousarray(own[idx])
        e.configure(G.make_config(lam, l0, ZG, psf=p, init=H.GUESS, **kw))
        return e.synthesize(np.ascontiguousarray(t[idx]))

    with G.Engine(0) as e:
        few = profiles(e, np.arange(n))
        assert np.isfinite(few).all()
        for count in (edge, edge + 1, edge + 2):
            idx = np.arange(count) % n
            np.testing.assert_array_equal(profiles(e, idx), few[idx], err_msg=str(count))
