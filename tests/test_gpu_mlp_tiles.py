"""Edges of the inference kernel's tiles and of its coalesced input rows: one
pixel, one short of a tile, a full one, one more, both slots of every CTA and
one pixel beyond, at grids whose rows fill part of a warp's lanes.  A pixel's
start model must not depend on where it lies, and must be the oracle's."""
import numpy as np
import pytest

import gmilos_b200 as G
import helpers as H
import mlp_oracle as M

pytestmark = pytest.mark.gpu

ZG = G.zeeman_from_levels(2, 1, 1.0, 2, 2, 0.0, 1.0)


@pytest.mark.parametrize("nl", [2, 9, 31, 32])
def test_start_models_at_tile_edges(nl):
    lam, _ = H.grid(nl)
    l0, _ = H.fe_line()
    net = H.random_net(40 + nl, nl)
    n = 2 * 148 * 128 + 1
    rng = np.random.default_rng(nl)
    obs = rng.normal(0.5, 0.2, (n, 4, nl)).astype(np.float32)
    obs[1000:2000] = obs[:1000]
    with G.Engine(0) as e:
        e.configure(G.make_config(lam, l0, ZG, init=H.GUESS))
        whole = e.mlp_predict(net, obs)
        np.testing.assert_array_equal(whole[1000:2000], whole[:1000])
        for k in (1, 127, 128, 129, 257):
            np.testing.assert_array_equal(e.mlp_predict(net, obs[:k]), whole[:k])
    p = M.params(net)
    idx = np.r_[0:300, n - 140:n]
    want, _ = M.predict(p, obs[idx], H.GUESS, H.FREE9)
    err = np.abs(M.targets(whole[idx]) - M.targets(want)) / p["out_scale"][:M.OUT]
    # as for the other inference tests: a few BF16 roundings of hidden activations may flip
    assert np.percentile(err, 99) < 5e-3 and np.median(err) < 5e-4


@pytest.mark.parametrize("nl,rows", [(32, 128), (30, 384), (9, 1152), (30, 148 * 128 + 128)])
def test_gradients_at_batch_edges(nl, rows):
    """Batches of one tile, of fewer 64-row steps than batch slices, of an odd
    number of tiles and of one tile more than the SMs: every weight and bias
    gradient is the oracle's to 1 % (as for the other gradient test), and a
    repeated call gives the same gradients bit for bit (partials summed in
    order)."""
    lam, _ = H.grid(nl)
    l0, _ = H.fe_line()
    net = H.random_net(70 + nl, nl)
    rng = np.random.default_rng(rows)
    truth = H.truth_models(rows, rng)
    obs = rng.normal(0.3, 0.2, (rows, 4, nl)).astype(np.float32)
    with G.Engine(0) as e:
        e.configure(G.make_config(lam, l0, ZG, init=H.GUESS))
        loss, g = e.mlp_gradients(net, obs, truth)
        _, again = e.mlp_gradients(net, obs, truth)
    p = M.params(net)
    lo, go = M.loss_and_grads(p, M.inputs(p, obs), M.standardised_targets(p, truth).astype(np.float32).astype(np.float64))
    assert loss == pytest.approx(lo, rel=1e-3)
    ga, gb = g.arrays(), again.arrays()
    for name in ("w1", "b1", "w2", "b2", "w3", "b3"):
        a = np.asarray(ga[name], dtype=np.float64)
        np.testing.assert_array_equal(ga[name], gb[name])
        a = a[:M.OUT] if name == "b3" else a
        assert np.linalg.norm(a - go[name]) < 1e-2 * np.linalg.norm(go[name]), name
