"""Training in one launch per epoch (k_mlp_epoch, mini-batches of up to
eight blocks on one thread block cluster) and beyond it: every update of a
run equals Adam's step, taken here in FP64, on the device's own gradient
(checked against the CPU reference elsewhere) of that mini-batch, for
clusters of every size, part-filled blocks and ragged last mini-batches.

Tolerance: the gradient's FP32 sums run in the shuffled order (1e-6
relative), which Adam's quotient turns into at most a few percent of lr
where a gradient is near its eps; over a run of updates at most lr / 10 in
any parameter and 1e-3 lr on average."""
import numpy as np
import pytest

from bookleaf_f90_gb300.closure import ClosureNet, init_params

pytestmark = pytest.mark.gpu

RUNS = [(1, 64, 2), (63, 64, 1), (64, 64, 2), (65, 64, 2), (150, 100, 3), (129, 192, 1),
        (300, 256, 2), (500, 300, 1), (384, 384, 1), (449, 448, 1), (513, 512, 1), (600, 513, 1)]


def _orders(n, epochs, seed):
    mask = (1 << 64) - 1
    r = (seed * 0x9E3779B97F4A7C15 + 1) & mask
    perm = list(range(n))
    for _ in range(epochs):
        for i in range(n - 1, 0, -1):
            r = (r + 0x9E3779B97F4A7C15) & mask
            z = ((r ^ (r >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = (z ^ (z >> 31)) % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        yield list(perm)


def _gradient(params, x, t):
    import ctypes as ct
    net = ClosureNet(params)
    g, loss = np.zeros(len(params), np.float32), ct.c_float(0)
    x, t = np.ascontiguousarray(x), np.ascontiguousarray(t)
    vp = lambda a: a.ctypes.data_as(ct.c_void_p)
    assert net.L.bl_mlp_gradient(net.handle, vp(x), vp(t), len(x), vp(g), ct.byref(loss)) == 0
    net.close()
    return g.astype(np.float64), loss.value


@pytest.mark.parametrize("n,batch,epochs", RUNS)
def test_updates_are_adams_steps(n, batch, epochs):
    rng = np.random.default_rng(n + batch)
    x = rng.normal(0, 1, (n, 10)).astype(np.float32)
    t = rng.normal(0, 1, (n, 2)).astype(np.float32)
    lr, seed = 1e-3, 5
    net = ClosureNet(init_params(3))
    losses = net.train(x, t, epochs=epochs, batch=batch, lr=lr, seed=seed)
    got = net.params()
    net.close()
    p = init_params(3).astype(np.float64)
    m, v, step = np.zeros_like(p), np.zeros_like(p), 0
    for order, loss in zip(_orders(n, epochs, seed), losses):
        total = 0.0
        for at in range(0, n, batch):
            rows = order[at:at + batch]
            g, part = _gradient(p.astype(np.float32), x[rows], t[rows])
            total += part * len(rows)
            step += 1
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            p = p - lr * (m / (1 - 0.9 ** step)) / (np.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
        assert abs(loss - total / n) <= 1e-4 * abs(total / n)
    off = np.abs(got - p)
    assert np.max(off) <= 0.1 * lr and np.mean(off) <= 1e-3 * lr, (np.max(off), np.mean(off))
