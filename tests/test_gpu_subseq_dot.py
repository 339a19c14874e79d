"""euclidean / scaled euclidean subsequence minima through the dot-product
filter: distances and first indices of the oracle's scan, at the edges of its
window tiles and shapelet groups and on data that stresses its bounds (exact
and repeated matches, constant stretches, periodic series, offsets, zeros)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import oracle as O  # noqa: E402
from wildboar_gb300.distance import pairwise_subsequence_distance  # noqa: E402


def _data(kind, rng, n, T, lens):
    X = np.cumsum(rng.standard_normal((n, T)), axis=1)
    S = [np.cumsum(rng.standard_normal(k)) for k in lens]
    if kind == "cut":  # exact matches, some twice
        S = [X[i % n, 1:1 + k].copy() for i, k in enumerate(lens)]
        X[:, T // 2:] = X[:, :T - T // 2]
    elif kind == "periodic":
        X = np.tile(np.round(rng.standard_normal((n, 7)), 1), (1, T // 7 + 1))[:, :T]
        S = [np.tile(X[i % n, :7], k // 7 + 1)[:k] for i, k in enumerate(lens)]
    elif kind == "constant":
        X[0] = 3.0
        X[1:, 5:T // 2] = -1.5
        S[0][:] = 3.0
    elif kind == "offset":
        X, S = X + 3e5, [s + 3e5 for s in S]
    elif kind == "tiny":
        X, S = X * 1e-160, [s * 1e-160 for s in S]
    elif kind == "zero":
        X[:, :] = 0.0
    return X, S


@pytest.mark.parametrize("metric", ["euclidean", "scaled_euclidean"])
@pytest.mark.parametrize("kind", ["walk", "cut", "periodic", "constant", "offset", "tiny", "zero"])
@pytest.mark.parametrize("T", [70, 263, 300, 600, 1100])
def test_minimum_and_first_index(metric, kind, T):
    rng = np.random.default_rng(T)
    # groups of 1, 3, 4 and 5 shapelets, a whole-series one, one per tile edge
    lens = [8] * 5 + [9, 16, 16, 16, 31, 32, 33, 33, 33, 33, 40, min(T, 64), min(T, 256), T]
    X, S = _data(kind, rng, 4, T, lens)
    d, i = pairwise_subsequence_distance(S, X, metric=metric, return_index=True)
    od, oi = O.subsequence(S, X, metric=metric)
    np.testing.assert_array_equal(i, oi)
    np.testing.assert_allclose(d, od, rtol=1e-12, atol=0)
