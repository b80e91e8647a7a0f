"""The one-launch training epoch (minibatches of up to 32 x 128 rows) and the
launch-per-step one (4224 rows) against a host replay of their steps: the public
gradient on the same rows in the training order, and Adam in FP32 numpy.

One step: the gradients are the same bits, Adam rounds a handful of times, and
the weights are below 1 in magnitude, so 2e-7 (three roundings).  Several steps:
a weight's last bit may round to another BF16 operand (2^-9 of it), and where a
gradient is smaller than that change Adam's step, which is about the learning
rate whatever the gradient's size, may differ: 1e-5 for all but 1% of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BETA1, BETA2, EPS = np.float32(0.9), np.float32(0.999), np.float32(1e-8)


def training_order(n, seed):
    """Fisher-Yates from splitmix64 of the object's seed."""
    mask = (1 << 64) - 1
    s = seed ^ 0x5DEECE66D
    order = list(range(n))
    for r in range(n - 1, 0, -1):
        s = (s + 0x9E3779B97F4A7C15) & mask
        z = s
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        j = (z ^ (z >> 31)) % (r + 1)
        order[r], order[j] = order[j], order[r]
    return np.array(order)


@pytest.mark.parametrize("samples, batch", [(300, 256), (420, 128), (700, 256), (2400, 1024),
                                            (4600, 4096), (9200, 4096), (4800, 4224), (9600, 4224)])
def test_epoch_equals_its_steps(cuda, samples, batch):
    g = cuda.gravity_init(1.0, 0.01)
    with cuda.CudaContext() as ctx, cuda.CudaCorrection(seed=3) as corr:
        ctx.generate_preset("globular_cluster", 20000, 1)
        corr.generate(ctx, g, 1.0, samples, 7)
        x, y, rows = corr.samples()
        w, scaling = corr.parameters()
        xs = (x - scaling[:10]) * scaling[10:20]
        ys = (y - scaling[40:43]) / scaling[43:46]
        n = rows - (rows // 16) // 128 * 128  # the last sixteenth validates
        steps = n // batch
        assert 1 <= steps <= 3
        order = training_order(n, 3)
        m, v = np.zeros_like(w), np.zeros_like(w)
        with cuda.CudaCorrection(seed=3) as single:
            for k in range(steps):
                single.set_parameters(w, scaling)
                at = order[k * batch:(k + 1) * batch]
                grad, _ = single.gradient(xs[at], ys[at])
                m = BETA1 * m + (np.float32(1) - BETA1) * grad
                v = BETA2 * v + (np.float32(1) - BETA2) * grad * grad
                b1 = np.float32(1) - BETA1 ** np.float32(k + 1)
                b2 = np.float32(1) - BETA2 ** np.float32(k + 1)
                w = w - np.float32(1e-3) * (m / b1) / (np.sqrt(v / b2) + EPS)
        train, _ = corr.train(1, batch, 1e-3)
        after, _ = corr.parameters()
    assert np.isfinite(train[0]) and train[0] > 0
    off = np.abs(after - w)
    if steps == 1:
        assert np.max(off) <= 2e-7
    else:
        assert np.mean(off > 1e-5) < 0.01
