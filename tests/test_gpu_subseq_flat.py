"""scaled euclidean subsequence minima of collections in which some series have
flat or zero-padded stretches, or lie far from 0: their pairs are left to the FP64
scan, by rows of one length and one series, beside series that are settled."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import oracle as O  # noqa: E402
from wildboar_gb300.distance import pairwise_subsequence_distance  # noqa: E402


# lengths up to 130 take the tiled scan, with one of 400 all take the plain one
@pytest.mark.parametrize("longest", [130, 400])
# windows without a bound in the flat series: some below and above the limit of
# kept windows, all
@pytest.mark.parametrize("stretch", [18, 24, 25, 26, 41, 200, 520])
@pytest.mark.parametrize("flat", [0.0, -2.5, 1e6])
def test_some_flat_series(longest, stretch, flat):
    rng = np.random.default_rng(stretch)
    T = 520
    X = np.cumsum(rng.standard_normal((9, T)), axis=1)
    for i in (0, 4, 8):
        at = rng.integers(0, T - stretch + 1)
        X[i, at:at + stretch] = flat
    X[6] += 1e5  # some hundred standard deviations from 0
    lens = [9, 17, 17, 17, 32, 33, 64, 64, longest]
    S = [np.cumsum(rng.standard_normal(k)) for k in lens]
    d, i = pairwise_subsequence_distance(S, X, metric="scaled_euclidean", return_index=True)
    od, oi = O.subsequence(S, X, metric="scaled_euclidean")
    np.testing.assert_array_equal(i, oi)
    np.testing.assert_allclose(d, od, rtol=1e-12, atol=0)


# every series at a level and of a size of its own: the bounds of one do not
# suffer from another's
@pytest.mark.parametrize("levels", [[0, 1e3, -1e6, 1e9], [0, 0, 0, 1e160], [1e-200, 1e200, 0, 1],
                                    [1e-300, 1e-160, 1e300, 1e308]])
@pytest.mark.parametrize("size", [1.0, 1e-3, 1e4])
def test_series_of_different_levels(levels, size):
    rng = np.random.default_rng(3)
    X = np.cumsum(rng.standard_normal((5, 300)), axis=1)
    for i, v in enumerate(levels):
        X[i] = X[i] * size + v if abs(v) < 1e100 else X[i] * (v / 1e3)
    S = [np.cumsum(rng.standard_normal(k)) for k in (9, 17, 17, 40, 200)]
    S.append(X[1, 50:90].copy())
    with np.errstate(all="ignore"):
        d, i = pairwise_subsequence_distance(S, X, metric="scaled_euclidean", return_index=True)
        od, oi = O.subsequence(S, X, metric="scaled_euclidean")
    np.testing.assert_array_equal(i, oi)
    np.testing.assert_allclose(d, od, rtol=1e-12, atol=0)
