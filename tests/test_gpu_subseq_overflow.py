"""Subsequence minima of values whose squares overflow: the scan keeps no window
of an infinite (or NaN) sum, so the index is 0 and the distance infinite unless
some window's sum is finite."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import oracle as O  # noqa: E402
from wildboar_gb300.distance import (  # noqa: E402
    paired_subsequence_distance, pairwise_subsequence_distance)


def _data(kind, T):
    rng = np.random.default_rng(T)
    X = 1e160 * (2.0 + rng.random((4, T)))
    S = [-1e160 * (2.0 + rng.random(k)) for k in (3, 8, 17, 40, T - 2)]
    if kind == "some":  # a finite window late in two of the series
        X[1, T - 20:T - 3] = S[2] * (1 + 1e-9)
        X[2, T - 9:T - 1] = S[1]
    elif kind == "offset":  # large values of a small range
        X = 1e160 * (1.0 + 1e-9 * rng.standard_normal((4, T)))
        S = [X[i % 4, 2:2 + len(s)] * (1 - 1e-7) for i, s in enumerate(S)]
    return X, S


@pytest.mark.parametrize("metric,params", [("euclidean", None), ("scaled_euclidean", None),
                                           ("dtw", {"r": 0.2}), ("ddtw", {"r": 0.2})],
                         ids=["euclidean", "scaled", "dtw", "ddtw"])
@pytest.mark.parametrize("kind", ["all", "some", "offset"])
@pytest.mark.parametrize("T", [45, 130])
def test_minimum_and_first_index(metric, params, kind, T):
    X, S = _data(kind, T)
    kw = {} if params is None else {"metric_params": params}
    with np.errstate(all="ignore"):
        d, i = pairwise_subsequence_distance(S, X, metric=metric, return_index=True, **kw)
        od, oi = O.subsequence(S, X, metric=metric, **kw)
        pd, pi = paired_subsequence_distance(S[:4], X, metric=metric, return_index=True, **kw)
    np.testing.assert_array_equal(i, oi)
    np.testing.assert_allclose(d, od, rtol=1e-12, atol=0)
    at = np.arange(4)
    np.testing.assert_array_equal(pi, np.asarray(oi)[at, at])
    np.testing.assert_allclose(pd, np.asarray(od)[at, at], rtol=1e-12, atol=0)
