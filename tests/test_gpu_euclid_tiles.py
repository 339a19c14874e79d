"""The euclidean matrix at the tile choices' edges against numpy's float64
sums in the same order."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from wildboar_gb300.distance import pairwise_distance  # noqa: E402


@pytest.mark.parametrize("nx,ny,L", [(1, 1, 1), (7, 9, 31), (8, 8, 32), (9, 17, 33), (300, 257, 40),
                                     (320, 256, 5), (1300, 1000, 64), (1281, 993, 33)])
def test_tiles_match_the_ordered_sum(nx, ny, L):
    rng = np.random.default_rng(nx)
    X, Y = rng.standard_normal((nx, L)), rng.standard_normal((ny, L))
    acc = np.zeros((nx, ny))
    for k in range(L):
        v = Y[None, :, k] - X[:, None, k]
        acc = acc + v * v
    np.testing.assert_array_equal(np.asarray(pairwise_distance(X, Y)).reshape(nx, ny),
                                  np.sqrt(acc))
    if nx > 1:
        sq = np.zeros((nx, nx))
        for k in range(L):
            v = X[None, :, k] - X[:, None, k]
            sq = sq + v * v
        np.testing.assert_array_equal(pairwise_distance(X), np.sqrt(sq))
