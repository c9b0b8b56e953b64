"""Sums over the batch in the surrogate's gradients: repeatable to the bit, exact where every operand and every
partial sum is a small integer (any misplaced row, column or split shows), and as accurate as their additions allow."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bf16(x):
    u = np.ascontiguousarray(x, dtype=np.float32).view(np.uint32).astype(np.uint64)
    return ((u + 0x7FFF + ((u >> 16) & 1)) >> 16 << 16).astype(np.uint32).view(np.float32)


def _split(g, sizes):
    out, o = [], 0
    for a, b in zip(sizes[:-1], sizes[1:]):
        out += [g[o:o + a * b].reshape(b, a), g[o + a * b:o + a * b + b]]
        o += a * b + b
    return out


# one to eight tiles of every width (64 columns: the input layer); 1, 8 or 16, and 38 to 128 ragged splits of the batch
@pytest.mark.parametrize("width,nout", [(128, 2), (256, 1), (384, 2), (512, 4)])
@pytest.mark.parametrize("n,batch", [(128, 128), (2048, 4096), (65536, 65536)])
def test_integer_sums_are_exact(width, nout, n, batch):
    """Integer weights, biases of 64 (SiLU is the identity and its derivative 1 there to the last bit), a permutation
    as the second layer, n and nout powers of two: every product and sum of the step is an integer (times 2 / (n nout))
    that FP32 and, where rounded, BF16 hold exactly."""
    from symboltz.surrogate import MLP
    rng = np.random.default_rng(width + n)
    nin = 9
    x = rng.integers(-2, 3, (n, nin)).astype(np.float64)
    e = rng.integers(-2, 3, (n, nout)).astype(np.float64)  # residuals
    W0 = rng.integers(-1, 2, (width, nin)).astype(np.float64)
    perm = rng.permutation(width)
    W1 = np.eye(width)[perm]
    W2 = rng.choice([-4.0, -2.0, -1.0, 1.0, 2.0, 4.0], (nout, width))
    X1 = x @ W0.T + 64
    X2 = X1[:, perm] + 64
    b2 = -np.round(X2.mean(0) @ W2.T)
    y = X2 @ W2.T + b2
    assert X1.min() > 32 and X2.max() < 256
    net = MLP(nin, width, 2, nout, batch, 1)
    net.set_params(np.concatenate([W0.ravel(), np.full(width, 64.0), W1.ravel(), np.full(width, 64.0), W2.ravel(), b2]).astype(np.float32))
    loss, g = net.gradients(x, y - e)
    sc = 2.0 / (n * nout)
    dZ2 = e @ W2
    dZ1 = np.zeros_like(dZ2)
    dZ1[:, perm] = dZ2
    assert np.abs(dZ2).max() < 256
    ref = [dZ1.T @ x, dZ1.sum(0), dZ2.T @ X1, dZ2.sum(0), e.T @ X2, e.sum(0)]
    assert max(np.abs(r).max() for r in ref) < 2.0 ** 22
    assert loss == pytest.approx(np.mean(e ** 2), rel=1e-13)
    for a, r in zip(_split(g.astype(np.float64), [nin, width, width, nout]), ref):
        np.testing.assert_array_equal(a, sc * r)


@pytest.mark.parametrize("width,nhidden,nout,batch", [(512, 3, 7, 65536), (256, 2, 1, 8192), (1024, 1, 64, 4096)])
def test_equal_trainings_give_equal_bits(width, nhidden, nout, batch):
    from symboltz.surrogate import MLP
    rng = np.random.default_rng(4)
    X = rng.uniform(-1, 1, (batch, 10)).astype(np.float32)
    Y = np.sin(3 * X @ rng.normal(size=(10, nout))).astype(np.float32)
    p0, runs = None, []
    for _ in range(3):
        net = MLP(10, width, nhidden, nout, batch, 1)
        p0 = net.get_params() if p0 is None else p0
        net.set_params(p0)
        loss0, g = net.gradients(X, Y)
        net.set_data(X, Y)
        runs.append((loss0, g, net.train(5, 1e-3), net.get_params()))
        assert not np.array_equal(runs[-1][3], p0)
    for r in runs[1:]:
        for a, b in zip(r, runs[0]):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n,batch", [(65536, 65536), (41088, 65536)])
def test_bias_sums_round_a_few_times(n, batch):
    """Positive terms: a tree over 32 rows rounds 5 times (256 rows of the output layer: 5, then 7 in a chain), the
    compensated sum of those parts about twice, each by at most 2^-24 of the sum."""
    from symboltz.surrogate import MLP
    rng = np.random.default_rng(n)
    width = 256
    x = rng.uniform(-1, 1, (n, 5)).astype(np.float32)
    t = -rng.uniform(0.5, 1.5, (n, 1)).astype(np.float32)
    W2 = rng.choice([0.25, 0.5, 1.0, 2.0], (1, width))
    net = MLP(5, width, 1, 1, batch, 1)
    # zero input layer: pre-activations 0, SiLU' 1/2, outputs 0
    net.set_params(np.concatenate([np.zeros(5 * width + width), W2.ravel(), [0.0]]).astype(np.float32))
    _, g = net.gradients(x, t)
    dy = _bf16(np.float32(2.0) / np.float32(n) * -t).astype(np.float64)
    _, b0, _, b1 = _split(g.astype(np.float64), [5, width, 1])
    ref = dy.sum()
    np.testing.assert_allclose(b1, ref, rtol=14 * 2.0 ** -24)
    np.testing.assert_allclose(b0, 0.5 * W2[0] * ref, rtol=7 * 2.0 ** -24)
