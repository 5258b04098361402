"""A ragged batch's captured device work against a change of configuration
between calls: free parameters, numerics, iteration limit, macroturbulence and
the number of terms.  A call with use_graph after gm_configure must give what
a direct call gives, bit for bit -- on the call that follows the change and on
the replay after it -- and so must the call after the change back."""
import numpy as np
import pytest

import gmilos_b200 as G
from gmilos_b200 import batch
import helpers as H
import oracle as O

pytestmark = pytest.mark.gpu

ZG = G.zeeman_from_levels(2, 1, 1.0, 2, 2, 0.0, 1.0)
L0 = 6173.3356
KEYS = ("model", "chi2", "iters", "status")
VMAC = H.GUESS[:9] + (0.8, 1.0)
CHANGES = {"fix": dict(fix=(1, 1, 1, 1, 0, 1, 1, 1, 1, 0, 0)), "one free": dict(fix=(0, 1) + (0,) * 9),
           "numerics": dict(numerics=1), "longer": dict(miter=19), "shorter": dict(miter=5),
           "quirks": dict(reference_quirks=0), "vmac": dict(init=VMAC),
           "eleven": dict(fix=(1,) * 11, init=VMAC), "noise": dict(noise=2e-3)}


def psf_for(lam):
    return O.psf_gauss(100.0, lam)


def config(**kw):
    lam, _ = H.grid(30)
    return G.make_config(lam, L0, ZG, **{**dict(init=H.GUESS, miter=12, noise=1e-3), **kw})


@pytest.fixture(scope="module")
def engine():
    e = G.Engine(0)
    yield e
    e.close()


@pytest.fixture(scope="module")
def rois(engine):
    rng = np.random.default_rng(77)
    out = []
    for side, nl in ((160, 30), (16, 45), (9, 12)):
        lam, _ = H.grid(nl)
        engine.configure(G.make_config(lam, L0, ZG, psf=psf_for(lam), init=H.GUESS))
        o = engine.synthesize(H.truth_models(side * side, rng))
        out.append((np.ascontiguousarray(o + rng.normal(0, 1e-3, o.shape).astype(np.float32)), lam))
    return out


def same(got, want):
    for g, w in zip(got, want):
        for k in KEYS:
            np.testing.assert_array_equal(g[k], w[k], err_msg=k)


@pytest.mark.parametrize("change", sorted(CHANGES))
def test_reconfigured_batches_equal_direct_calls(engine, rois, change):
    first, second = config(), config(**CHANGES[change])
    want = []
    for c in (first, second):
        engine.configure(c)
        want.append(batch.invert_rois(engine, rois, psf_for)[0])
    # the quirk is one of the filling factor's derivative, and batches have no stray light
    assert change == "quirks" or any((a["model"] != b["model"]).any() for a, b in zip(*want)), "the change changes nothing"
    for c, w in ((first, want[0]), (second, want[1]), (first, want[0])):
        engine.configure(c)
        for replay in (0, 1):
            got, st = batch.invert_rois(engine, rois, psf_for, use_graph=True)
            same(got, w)
            if replay:
                assert st["graph_replayed"] == 1


@pytest.mark.parametrize("kw", [dict(), dict(init=VMAC), dict(fix=(1,) * 11, init=VMAC)], ids=["ten", "vmac", "eleven"])
@pytest.mark.parametrize("some", [(0, 1, 2), (1, 2), (2,)])
def test_a_replay_reports_the_launches_it_runs(engine, rois, kw, some):
    engine.configure(config(**kw))
    part = [rois[i] for i in some]
    counts = []
    for use_graph in (False, True, True):
        _, st = batch.invert_rois(engine, part, psf_for, use_graph=use_graph)
        counts.append(st["launches"])
        assert engine.stats()["kernel_launches"] == st["launches"]
    assert st["graph_replayed"] == 1
    # every wave has a trial kernel, all but the last an accept kernel, and a class a pre-pass
    assert counts[0] == counts[1] == counts[2] >= (1 + 2 * 13 - 1) * (1 if len(some) == 1 else 2)


def test_the_solve_kernel_of_large_batches_changes_nothing(engine, rois):
    """A class of 12 288 pixels and more makes its steps in a kernel of its own:
    regions alone on either side of that, in 10 terms with and without
    macroturbulence, at one and two samples per lane, equal those in a batch
    beyond it, bit for bit."""
    lam45, _ = H.grid(45)
    obs, lam = rois[0]
    few, _ = rois[1]
    wide = np.ascontiguousarray(np.tile(few, (50, 1, 1))[:12288])
    for kw in (dict(), dict(init=VMAC), dict(numerics=1), dict(logclambda=1), dict(fix=(0, 1) + (0,) * 9)):
        engine.configure(config(**kw))
        for cube, grid in ((obs[:12288], lam), (wide, lam45)):
            whole, large = batch.invert_rois(engine, [(cube, grid)], psf_for)
            part, small = batch.invert_rois(engine, [(np.ascontiguousarray(cube[:12287]), grid)], psf_for)
            assert large["launches"] == 1 + 3 * 13 - 2 and small["launches"] == 1 + 2 * 13 - 1
            for k in KEYS:
                np.testing.assert_array_equal(whole[0][k][:12287], part[0][k], err_msg=k)
