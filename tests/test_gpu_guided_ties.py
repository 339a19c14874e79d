"""Guided evaluation of values that tie everywhere, with more tiles than warps:
the later tiles go to the full recurrence at once, with the same bits."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from wildboar_gb300.distance import paired_distance, pairwise_distance  # noqa: E402


@pytest.mark.parametrize("metric,r", [("dtw", 0.3), ("dtw", 1.0), ("adtw", 0.5), ("wdtw", 1.0)])
@pytest.mark.parametrize("kind", ["binary", "spike", "constant"])
@pytest.mark.parametrize("same", [False, True])
def test_same_bits_as_the_ring_kernel(metric, r, kind, same, monkeypatch):
    rng = np.random.default_rng(1)

    def data(n, length):
        if kind == "binary":
            return (rng.random((n, length)) > 0.5).astype(float)
        if kind == "spike":
            return (np.arange(length)[None, :] == rng.integers(0, length, (n, 1))).astype(float)
        return np.ones((n, length))

    X = data(520 if same else 320, 104)
    args = (X,) if same else (X, data(331, 120))
    monkeypatch.delenv("WB_GPU_ELASTIC", raising=False)
    got = pairwise_distance(*args, metric=metric, metric_params={"r": r})
    monkeypatch.setenv("WB_GPU_ELASTIC", "ring")
    np.testing.assert_array_equal(
        got, pairwise_distance(*args, metric=metric, metric_params={"r": r}))


@pytest.mark.parametrize("metric,r", [("dtw", 0.1), ("dtw", 1.0), ("adtw", 0.4), ("wdtw", 1.0)])
@pytest.mark.parametrize("lx,ly", [(100, 100), (330, 130), (130, 331), (600, 610)])
def test_few_pairs_left(metric, r, lx, ly, monkeypatch):
    """Some pairs of constant series among walks: left over one by one."""
    rng = np.random.default_rng(lx)
    X = np.cumsum(rng.standard_normal((37, lx)), axis=1)
    Y = np.cumsum(rng.standard_normal((21, ly)), axis=1)
    X[3] = X[17] = 1.0
    Y[5] = Y[20] = 1.0
    X[8] = np.round(X[8] / 8)
    monkeypatch.delenv("WB_GPU_ELASTIC", raising=False)

    def calls():
        out = [pairwise_distance(X, Y, metric=metric, metric_params={"r": r}),
               pairwise_distance(X, metric=metric, metric_params={"r": r})]
        if lx == ly:
            out.append(paired_distance(X[:21], Y, metric=metric, metric_params={"r": r}))
        return out

    got = calls()
    monkeypatch.setenv("WB_GPU_ELASTIC", "ring")
    for a, b in zip(got, calls()):
        np.testing.assert_array_equal(a, b)
