"""dtw / ddtw subsequence minima through the float32 window filter: distances
and first indices of the oracle's scan, at the edges of the filter's register
blocks (half-widths), its window rounds and its kept-window lists (ties,
periodic and constant series), pairwise and paired."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import oracle as O  # noqa: E402
from wildboar_gb300.distance import (  # noqa: E402
    paired_subsequence_distance, pairwise_subsequence_distance)


def _data(kind, rng, n, T, lens):
    X = np.cumsum(rng.standard_normal((n, T)), axis=1)
    S = [np.cumsum(rng.standard_normal(k)) for k in lens]
    if kind == "cut":  # exact matches, some twice
        S = [X[i % n, 3:3 + k].copy() for i, k in enumerate(lens)]
        X[:, T // 2:] = X[:, :T - T // 2]
    elif kind == "periodic":
        X = np.tile(np.round(rng.standard_normal((n, 7)), 1), (1, T // 7 + 1))[:, :T]
        S = [np.tile(X[i % n, :7], k // 7 + 1)[:k] for i, k in enumerate(lens)]
    elif kind == "constant":
        X = np.full((n, T), 2.5)
    elif kind == "offset":
        X, S = X + 1e7, [s + 1e7 for s in S]
    elif kind == "tiny":
        X, S = X * 1e-160, [s * 1e-160 for s in S]
    return X, S


@pytest.mark.parametrize("metric", ["dtw", "ddtw"])
@pytest.mark.parametrize("kind", ["walk", "cut", "periodic", "constant", "offset", "tiny"])
@pytest.mark.parametrize("r", [0.02, 0.1, 0.25, 0.5])
def test_minimum_and_first_index(metric, kind, r):
    rng = np.random.default_rng(int(r * 100))
    lens = [3, 16, 31, 32, 33, 63, 64, 90]
    X, S = _data(kind, rng, 5, 160, lens)
    kw = dict(metric=metric, metric_params={"r": r}, return_index=True)
    d, i = pairwise_subsequence_distance(S, X, **kw)
    od, oi = O.subsequence(S, X, metric=metric, metric_params={"r": r})
    np.testing.assert_array_equal(i, oi)
    np.testing.assert_allclose(d, od, rtol=1e-12, atol=0)
    d, i = paired_subsequence_distance(S[:5], X, **kw)
    np.testing.assert_array_equal(i, np.asarray(oi)[np.arange(5), np.arange(5)])
    np.testing.assert_allclose(d, np.asarray(od)[np.arange(5), np.arange(5)], rtol=1e-12, atol=0)
