"""Training data that the default stream is still writing: gm_mlp_train and
gm_mlp_gradients, which run on the context's stream, take it as it will be."""
import numpy as np
import pytest

import gmilos_b200 as G
import helpers as H

pytestmark = pytest.mark.gpu

ZG = G.zeeman_from_levels(2, 1, 1.0, 2, 2, 0.0, 1.0)


@pytest.mark.parametrize("nl,rows", [(30, 1024), (9, 70016)])
def test_training_waits_for_the_default_stream(nl, rows):
    torch = pytest.importorskip("torch")
    lam, _ = H.grid(nl)
    l0, _ = H.fe_line()
    rng = np.random.default_rng(nl)
    truth = torch.from_numpy(H.truth_models(rows, rng)).cuda()
    obs = torch.from_numpy(rng.normal(0.4, 0.2, (rows, 4, nl)).astype(np.float32)).cuda()
    late_obs, late_truth = torch.zeros_like(obs), torch.zeros_like(truth)
    torch.cuda.synchronize()

    def late():
        torch.cuda.synchronize()
        late_obs.zero_()
        late_truth.zero_()
        torch.cuda._sleep(50_000_000)   # some 25 ms on the default stream
        late_obs.copy_(obs)
        late_truth.copy_(truth)
        return late_obs, late_truth

    with G.Engine(0) as e:
        e.configure(G.make_config(lam, l0, ZG, init=H.GUESS))
        want, got = G.mlp_new(nl, 5), G.mlp_new(nl, 5)
        loss = e.mlp_train(want, obs, truth, epochs=1, batch=512)
        assert np.all(np.isfinite(loss)) and want.arrays()["in_scale"][0] > 0
        e.mlp_train(got, *late(), epochs=1, batch=512)
        for k, v in want.arrays().items():
            if k in ("in_mean", "in_scale", "out_mean", "out_scale"):
                np.testing.assert_array_equal(got.arrays()[k], v, err_msg=k)
        l1, g1 = e.mlp_gradients(want, obs[:512], truth[:512])
        a, b = late()
        l2, g2 = e.mlp_gradients(want, a[:512], b[:512])
        for k, v in g1.arrays().items():
            np.testing.assert_array_equal(g2.arrays()[k], v, err_msg=k)
