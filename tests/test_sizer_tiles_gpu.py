"""The sizer's kernels where their tiles end (16, 32 and 64 samples; one more
than a round of CTAs) against the float64 statement of the network."""
import numpy as np
import pytest

from gpudbmetalcodegen_b200 import batch as B
from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 15, 16, 17, 33, 512, 32 * 148 - 1, 32 * 148, 32 * 148 + 31, 64 * 148 - 1, 64 * 148, 64 * 296 + 1, 40_003]


@pytest.mark.parametrize("n", SIZES)
def test_gradients_and_outputs(n):
    rng = np.random.default_rng(n)
    X = rng.random((n, 16), dtype=np.float32)
    Y = rng.random((n, 2), dtype=np.float32)
    s = B.Sizer(seed=n)
    p = s.params
    loss, g = M.loss_and_grads(p, X, Y)
    y, _ = M.forward(p, X)
    got, l = s.grads(X, Y)
    # FP32: a dot of 64 terms and a sum over n samples, each add 2^-24 off
    tol = (64 + np.sqrt(n)) * 2.0**-24
    assert abs(l - loss) <= 4 * tol * loss
    at = 0
    for name, shape in M.SHAPES:
        k = int(np.prod(shape))
        # ReLU masks of activations within rounding of zero may differ
        assert np.abs(got[at:at + k] - g[at:at + k]).max() <= 2e-3 * np.abs(g[at:at + k]).max(), name
        at += k
    assert np.linalg.norm(got - g) <= 50 * tol * np.linalg.norm(g)
    assert np.abs(s.predict(X) - y).max() <= 8 * 64 * 2.0**-24 * np.abs(y).max()
    s.close()
