"""The order of the learned guess' calls.  Training data that the default
stream is still writing: gm_mlp_train and gm_mlp_gradients, which run on the
context's stream, take it as it will be.  The network that gm_mlp_predict keeps
on the device: edited in place, exchanged for another of the same grid, trained
or differentiated between two calls, on changing streams, every call gives what
a context of its own gives."""
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


def test_predictions_follow_the_network():
    torch = pytest.importorskip("torch")
    nl, n = 30, 5000
    lam, _ = H.grid(nl)
    l0, _ = H.fe_line()
    rng = np.random.default_rng(3)
    obs = rng.normal(0.4, 0.2, (n, 4, nl)).astype(np.float32)
    truth = H.truth_models(n, rng)
    dev = torch.from_numpy(obs).cuda()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    cfg = G.make_config(lam, l0, ZG, init=H.GUESS)

    def alone(net):
        with G.Engine(0) as e:
            e.configure(cfg)
            return e.mlp_predict(net, obs)

    def on_stream(e, net, k):
        out = torch.empty((n, G.NPAR), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        G._check(G.lib().gm_mlp_predict(e._ctx, G.C.byref(net), G._ptr(dev), n, G._ptr(out),
                                        G.C.c_void_p(streams[k].cuda_stream)), e._ctx)
        return out.cpu().numpy()

    a, b = H.random_net(1, nl), H.random_net(2, nl)
    with G.Engine(0) as e:
        e.configure(cfg)
        for net in (a, b, a):
            np.testing.assert_array_equal(e.mlp_predict(net, obs), alone(net))
        a.arrays()["b3"][3] += 0.25
        np.testing.assert_array_equal(e.mlp_predict(a, obs), alone(a))
        e.mlp_gradients(b, obs[:256], truth[:256])
        np.testing.assert_array_equal(e.mlp_predict(a, obs), alone(a))
        e.mlp_train(b, obs, truth, epochs=1, batch=512)
        for net in (a, b):
            np.testing.assert_array_equal(e.mlp_predict(net, obs), alone(net))
        for k, net in enumerate((a, b, a, b)):
            np.testing.assert_array_equal(on_stream(e, net, (k // 2) & 1), alone(net))


def test_the_training_workspace_makes_room():
    """The workspace that stays with the context is given back when another
    allocation fails (one of 352 GB here, refused at once), and is made again by
    the next training call."""
    torch = pytest.importorskip("torch")
    nl, n = 30, 16384
    lam, _ = H.grid(nl)
    l0, _ = H.fe_line()
    rng = np.random.default_rng(8)
    truth = torch.from_numpy(H.truth_models(n, rng)).cuda()
    obs = torch.from_numpy(rng.normal(0.4, 0.2, (n, 4, nl)).astype(np.float32)).cuda()
    model = np.zeros((1, 11))
    out = np.zeros((1, 4, nl), np.float32)
    with G.Engine(0) as e:
        e.configure(G.make_config(lam, l0, ZG, init=H.GUESS))
        net = G.mlp_new(nl, 5)
        e.mlp_train(net, obs, truth, epochs=1, batch=n)
        kept = torch.cuda.mem_get_info()[0]
        with pytest.raises(G.GmError):
            G._check(G.lib().gm_synthesize_f64(e._ctx, G._ptr(model), 4_000_000_000, G._ptr(out), None, None), e._ctx)
        # 3.5 KB a row of the batch
        assert torch.cuda.mem_get_info()[0] - kept > 3000 * n
        loss = e.mlp_train(net, obs, truth, epochs=1, batch=n)
        assert np.isfinite(loss).all()
