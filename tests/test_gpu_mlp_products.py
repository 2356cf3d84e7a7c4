"""The network's gradients where every product is exact, against FP64.

Small integers in, two weights of +-1 per unit, and biases that hold the hidden
pre-activations at 18 and above, where SiLU is the identity in FP32 (sigmoid
rounds to 1): every activation is an integer of at most 256 (exact in BF16),
every output gradient a small integer times a power of two, and every sum stays
below 2^24.  So the gradients have to be equal, whatever tile shape and ring
depth the sizes select and however the weight gradients share a launch (up to
eight layers do); the bias gradients are sums of the same exact terms."""
import numpy as np
import pytest

from gundam_gb300.surrogate import MLP

pytestmark = pytest.mark.gpu

SIZES = [
    # dims, rows: what they select
    ([16, 72, 200, 8], 8),  # 32-column tiles, a few of them partial
    ([24] * 10 + [16], 32),  # ten layers: two launches of weight gradients
    ([200, 512, 512, 1024], 256),  # weight gradients in 64-column tiles
    ([40, 136, 8], 2048),  # narrow outputs
    ([200, 512, 512, 512, 2048], 1024),  # loss in 128-column tiles
    ([200, 512, 512, 512, 4096], 2048),  # loss in 64-column tiles, weight gradients in 128-column ones
    ([104, 512, 8192], 2048),  # loss in 256-column tiles
]


@pytest.mark.parametrize("dims,rows", SIZES)
def test_integer_gradients_are_exact(dims, rows):
    rng = np.random.default_rng(5)
    L = len(dims) - 1
    x = rng.integers(-8, 9, (rows, dims[0])).astype(np.float32)
    net = MLP(dims, batch_max=rows)
    ws, hs, h = [], [x], x
    for l in range(L):
        w = np.zeros((dims[l + 1], dims[l]), dtype=np.float32)
        unit = np.arange(dims[l + 1])
        w[unit, rng.permutation(dims[l + 1]) % dims[l]] = 1
        if l < 2 or l == L - 1:
            w[unit, rng.permutation(dims[l + 1]) % dims[l]] -= 1
        b = np.full(dims[l + 1], 64 if l < min(2, L - 1) else 0, dtype=np.float32)
        net.set_layer(l, w, b)
        h = h @ w.T + b
        assert np.abs(h).max() <= 256 and (l == L - 1 or h.min() >= 18)
        ws.append(w)
        hs.append(h)
    r = rng.integers(-2, 3, h.shape).astype(np.float32)
    gw, gb, loss = net.gradients(x, h + r)
    unit = 2.0 / (rows * dims[-1])  # a power of two
    dz = -r
    for l in range(L - 1, -1, -1):
        assert np.abs(dz).max() <= 256
        assert np.array_equal(gw[l], (dz.T @ hs[l]) * np.float32(unit)), l
        assert np.array_equal(gb[l], dz.sum(axis=0) * np.float32(unit)), l
        dz = dz @ ws[l]
    # one FP32 sum of rows * dims[-1] exact squares and its atomic adds
    assert abs(loss - np.mean(r.astype(np.float64) ** 2)) <= 1e-5
    net.close()
