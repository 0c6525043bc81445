"""Every tensor of the training and calibration kernels by itself against the
numpy restatement, over several batches of an epoch too, and what must not
change bit for bit.

A gradient that is missing or of another parameter moves a weight by another
lr a step or by none: a share of 1 of lr x steps.  The kernels' tanh.approx
(a BF16 unit, 2^-8, here and there) turns the sign of Adam's first steps where
a gradient is small against that: a few weights in a thousand, a share of 0.1
of a matrix; of 32 biases one or two, 0.35 to 0.5."""
import numpy as np
import pytest

from sph_gb300 import LearnedModel, Simulation
from test_gpu_learned import act_bf16, bf16
from test_gpu_training import act_grad, still_fluid

pytestmark = pytest.mark.gpu

GOLDEN, M64 = 0x9E3779B97F4A7C15, (1 << 64) - 1
MATRIX, VECTOR = 0.1, 0.5


def rnd(v):
    return bf16(np.asarray(v, np.float32)).astype(np.float64)


def shuffled(n, seed, adam_t, epochs):
    """The sample orders of a training call (splitmix64, Fisher-Yates)."""
    order, rng, out = list(range(n)), (seed * GOLDEN + 17 + adam_t) & M64, []
    for _ in range(epochs):
        for i in range(n - 1, 0, -1):
            rng = (rng + GOLDEN) & M64
            z = rng
            z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M64
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M64
            j = (z ^ (z >> 31)) % (i + 1)
            order[i], order[j] = order[j], order[i]
        out.append(np.array(order))
    return out


def train(w, x, target, batches, lr, outputs, trunk):
    """Adam steps on the given batches of samples; `outputs` in the loss."""
    p = {k: v.astype(np.float64).copy() for k, v in LearnedModel.unpack(w).items()}
    m, v = ({k: np.zeros_like(q) for k, q in p.items()} for _ in range(2))
    losses = []
    for t, b in enumerate(batches, 1):
        q = {k: rnd(a) for k, a in p.items()}
        z1 = x[b] @ q["W1"].T + q["b1"]
        h1 = act_bf16(z1)
        z2 = h1 @ q["W2"].T + q["b2"]
        h2 = act_bf16(z2)
        d = (h2 @ q["W3"].T + p["b3"])[:, outputs] - target[b]
        losses.append(float((d * d).sum()) / len(b))
        dy = np.zeros((len(b), LearnedModel.OUT))
        dy[:, outputs] = rnd(2.0 * d / len(b))
        g = dict(W3=dy.T @ h2, b3=dy.sum(0))
        if trunk:
            dz2 = rnd((dy @ q["W3"]) * act_grad(z2))
            dz1 = rnd((dz2 @ q["W2"]) * act_grad(z1))
            g.update(W1=dz1.T @ x[b], W2=dz2.T @ h1, b2=dz2.sum(0))
        for k in g:
            m[k] = 0.9 * m[k] + 0.1 * g[k]
            v[k] = 0.999 * v[k] + 0.001 * g[k] ** 2
            p[k] -= lr * (m[k] / (1 - 0.9 ** t)) / (np.sqrt(v[k] / (1 - 0.999 ** t)) + 1e-8)
    return p, losses


def share(got, want, scale):
    return np.sqrt(np.mean(((got - want) / scale) ** 2))


def eligible(sc, count):
    """Particles of few enough neighbours, in the order of their slots."""
    key = np.floor(sc.y).astype(np.int64) * sc.size_x + np.floor(sc.x).astype(np.int64)
    order = np.argsort(key, kind="stable")
    return order[(count[order] >= 0) & (count[order] <= LearnedModel.MAX_NEIGHBORS)]


@pytest.mark.parametrize("tiles,batch,epochs", [(1, 128, 3), (3, 384, 3), (6, 256, 2), (160, 2560, 1)])
def test_each_tensor_of_a_training_call(cuda_lib, tiles, batch, epochs):
    rows, lr, seed = 128 * tiles, 1e-3, 6
    sc = still_fluid(rows + 700, seed=50 + tiles)
    P = sc.params
    with Simulation.from_scene(sc) as s, LearnedModel(rows, seed=seed) as m:
        f, count = s.learned_features()
        dx, dy = s.probe_relaxation(P.as_dict())
        assert m.collect(s) == rows
        w0 = m.get_params() + np.random.default_rng(8).normal(0.0, 0.02, m.num_params()).astype(np.float32)
        m.set_params(w0)
        loss = m.train(epochs, batch, lr)
        w = m.get_params()
    take = eligible(sc, count)[:rows]
    scale = P.smoothing_radius * P.time_step ** 2 * (P.k + P.k_near + P.k_spring)
    target = np.stack([dx, dy], 1)[take].astype(np.float64) / scale
    orders = shuffled(rows, seed, 0, epochs)
    batches = [o[b:b + batch] for o in orders for b in range(0, rows, batch)]
    ref, losses = train(w0, f[take].astype(np.float64), target, batches, lr, [0, 1], True)
    assert np.isclose(loss, np.mean(losses[-(rows // batch):]), rtol=2e-2)
    got, was, unit = LearnedModel.unpack(w), LearnedModel.unpack(w0), lr * len(batches)
    assert np.array_equal(got["b1"], was["b1"])  # acts through the constant feature
    assert np.array_equal(got["W3"][2:], was["W3"][2:]) and np.array_equal(got["b3"][2:], was["b3"][2:])
    shares = {k: share(got[k], ref[k], unit) for k in ("W1", "W2")}
    shares["W3"] = share(got["W3"][:2], ref["W3"][:2], unit)
    assert max(shares.values()) <= MATRIX, shares
    small = {f"b2[{32 * k}:]": share(got["b2"][32 * k:32 * k + 32], ref["b2"][32 * k:32 * k + 32], unit)
             for k in range(4)}
    small["b3"] = share(got["b3"][:2], ref["b3"][:2], unit)
    assert max(small.values()) <= VECTOR, small


def densities(px, py, h):
    """Densities at given positions, each over all the others."""
    out = np.zeros(len(px))
    for i in range(len(px)):
        r = np.sqrt((px - px[i]) ** 2 + (py - py[i]) ** 2) / h
        r[i] = 1.0
        out[i] = np.sum(np.where(r < 1.0, 1.0 - r, 0.0) ** 2)
    return out


def test_calibration_trains_the_error_output_alone(cuda_lib):
    rows, lr, epochs = 1024, 1e-3, 3
    sc = still_fluid(rows, seed=77)
    P = sc.params
    with Simulation.from_scene(sc) as s, LearnedModel(rows, seed=3) as m:
        f, count = s.learned_features()
        assert np.all((count >= 0) & (count <= LearnedModel.MAX_NEIGHBORS))  # one batch: all of them
        w0 = m.get_params()
        scale = P.smoothing_radius * P.time_step ** 2 * (P.k + P.k_near + P.k_spring)
        net = m.forward(f)[:, :2].astype(np.float64) * scale
        plain = np.stack(s.probe_relaxation(P.as_dict()), 1).astype(np.float64)
        loss = m.calibrate(s, epochs, lr)
        w = m.get_params()
        assert m.num_samples == 0
    x = np.stack([sc.x, sc.y], 1).astype(np.float64)
    rho = [densities(*(x + d).T, P.smoothing_radius) for d in (net, plain)]
    target = np.minimum(np.abs(rho[0] - rho[1]) / P.rest_density * 100.0, 10.0)[:, None]
    ref, losses = train(w0, f.astype(np.float64), target, [np.arange(rows)] * epochs, lr, [2], False)
    assert np.isclose(loss, losses[-1], rtol=2e-2)
    got, was = LearnedModel.unpack(w), LearnedModel.unpack(w0)
    for k in ("W1", "b1", "W2", "b2"):
        assert np.array_equal(got[k], was[k]), k
    others = [o for o in range(LearnedModel.OUT) if o != 2]
    assert np.array_equal(got["W3"][others], was["W3"][others])
    assert np.array_equal(got["b3"][others], was["b3"][others])
    assert share(got["W3"][2], ref["W3"][2], lr * epochs) <= MATRIX
    assert share(got["b3"][2], ref["b3"][2], lr * epochs) <= VECTOR
