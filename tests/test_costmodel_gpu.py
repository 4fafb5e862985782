"""The cost model's kernels at the edges of their tiles (16 samples, 4 rows and
samples per thread, two blocks per SM), against the float64 restatement
(oracle/mlp.py)."""
import threading

import numpy as np
import pytest

from symboliclib_gb300 import native

import oracle.mlp as omlp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,inputs,hidden", [(1, 1, 1), (15, 3, 5), (16, 4, 32), (17, 50, 33), (2500, 50, 64),
                                             (4865, 7, 64), (6000, 111, 110), (300, 256, 48)])
def test_gradient_and_prediction_at_tile_edges(n, inputs, hidden):
    """Norm-wise: FP32 chains of up to 256 + 2 x 110 terms (2^-24 each, 2e-5
    if all err one way) and, at thousands of samples, single samples whose
    ReLU argument rounds to the other side of zero (1 / n of a column each)."""
    rng = np.random.default_rng(n + inputs)
    X = rng.standard_normal((n, inputs)).astype(np.float32)
    y = rng.standard_normal(n).astype(np.float32)
    net = native.MLP(inputs, hidden, seed=3)
    p = net.params()
    g, loss = net.gradient(X, y)
    ref, ref_loss = omlp.gradient(p, X, y, inputs, hidden)
    assert np.linalg.norm(g - ref) <= 1e-4 * np.linalg.norm(ref)
    assert abs(loss - ref_loss) <= 1e-4 * ref_loss
    pred, _ = omlp.forward(p, X, inputs, hidden)
    assert np.linalg.norm(net.predict(X) - pred) <= 1e-4 * np.linalg.norm(pred)


def test_layers_beyond_a_blocks_share_are_refused():
    net = native.MLP(4, 128, seed=1)  # 128 x 128 weights: 64 KB
    with pytest.raises(RuntimeError):
        net.predict(np.zeros((8, 4), np.float32))


def test_networks_of_several_sizes_on_several_threads():
    """The shared memory that a launch may have is a property of the kernel, not
    of the network."""
    def work(inputs, hidden, out):
        rng = np.random.default_rng(inputs)
        X, y = rng.standard_normal((40, inputs)).astype(np.float32), rng.standard_normal(40).astype(np.float32)
        try:
            net = native.MLP(inputs, hidden, seed=3)
            first = net.gradient(X, y)[0]
            out.append(all(np.array_equal(net.gradient(X, y)[0], first) for _ in range(400)))
        except RuntimeError as e:
            out.append(str(e))
    results = [[] for _ in range(4)]
    threads = [threading.Thread(target=work, args=(*shape, out))
               for shape, out in zip([(50, 64), (111, 110), (256, 48), (20, 96)], results)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert results == [[True]] * 4


@pytest.mark.parametrize("n", [16, 17, 40])
def test_gradients_beyond_the_range_are_infinite(n):
    """One sample whose activations overflow, in a full tile and in ragged ones:
    sums with one infinity are infinite, not NaN."""
    X = np.ones((n, 1), np.float32)
    X[-1] = 3e38
    net = native.MLP(1, 1, seed=1)
    net.set_params(np.array([2, 0, 1, 0, 1, 0], np.float32))  # W1 b1 W2 b2 W3 b3
    g, loss = net.gradient(X, np.zeros(n, np.float32))
    assert np.all(g == np.inf) and loss == np.inf
