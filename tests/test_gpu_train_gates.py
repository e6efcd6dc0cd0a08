"""A nearly closed update gate of the training recurrences, to the relative
accuracy of FP32: with z = sigmoid(x) of an exactly given x below -18 the
gradient of z's bias is z times a factor that does not depend on x (1 - z
rounds to 1), so the gradients at x and at x0 = -24 have the ratio z(x) / z(x0).

Tolerance: exp within 1 ulp (1.2e-7), 1 + e and the quotient within half an ulp
each, four more roundings of 2^-24 on the way to the gradient (units whose two
terms have one sign: no cancellation): 4.8e-7 a run, 1e-6 for the two."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_closed_gate_is_relatively_accurate():
    import torch
    from trajsimimeasures_b200.engine import TrajSet
    from trajsimimeasures_b200.surrogate import Encoder
    rng = np.random.default_rng(5)
    s = TrajSet.from_lists([np.array([[0.0, 0.0]]), np.array([[1.0, 0.5]])])
    enc = Encoder.init(s, seed=1)
    sizes = {"w1": 640, "b1": 64, "wih": 384 * 64, "bih": 384, "whh": 384 * 128, "bhh": 384}
    at = dict(zip(sizes, np.cumsum([0] + list(sizes.values())[:-1])))
    p = enc.params.cpu().numpy().copy()
    for k, n in sizes.items():
        p[at[k]:at[k] + n] = 0
    p[at["w1"]:at["w1"] + 640] = rng.normal(0, 1, 640)
    p[at["b1"]:at["b1"] + 64] = rng.normal(0, 0.1, 64)
    p[at["wih"] + 256 * 64:at["wih"] + 384 * 64] = rng.normal(0, 0.3, 128 * 64)  # the rows of n alone
    x = rng.uniform(-70, -20, 128).astype(np.float32)
    z = slice(at["bih"] + 128, at["bih"] + 256)
    n = slice(at["bih"] + 256, at["bih"] + 384)

    def grad(v):
        p[z] = v
        enc.params.copy_(torch.from_numpy(p))
        g = enc.loss_grad(s, [0, 1], [0], [1], [0.3])[1].cpu().numpy().astype(np.float64)
        enc.check_training()
        return g[z], g[n]
    (g0, gn0), (g1, gn1) = grad(np.full(128, -24, np.float32)), grad(x)
    assert np.array_equal(gn0, gn1)  # what does not depend on z is the same to the bit
    # the two trajectories' n, in FP64: units where they differ in sign
    def bf(a):
        return torch.from_numpy(a).bfloat16().double().numpy()
    w1 = bf(p[at["w1"]:at["w1"] + 640]).reshape(64, 2, 5)[:, :, 2]
    xy = (s.pts.cpu().numpy().astype(np.float64) - enc.nrm[:2]) * enc.nrm[2:]
    a = np.maximum(p[at["b1"]:at["b1"] + 64] + xy @ w1.T, 0)
    nn = np.tanh(a @ bf(p[at["wih"] + 256 * 64:at["wih"] + 384 * 64]).reshape(128, 64).T)
    ok = (nn[0] * nn[1] < -0.01) & (g0 != 0)
    assert ok.sum() >= 20
    sig = lambda v: 1.0 / (1.0 + np.exp(-v.astype(np.float64)))  # noqa: E731
    err = np.abs(g1[ok] / g0[ok] / (sig(x[ok]) / sig(np.array([-24.0]))) - 1)
    assert err.max() < 1e-6, err.max()
