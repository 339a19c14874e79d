"""Guided evaluation of collections that tie everywhere, or partly: rows that do
not fill a tile, a few tied series among others, tied series in a few rows.  Their
pairs go to the full recurrence before, within and after the guided kernel's tiles,
with the same bits."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from wildboar_gb300.distance import argmin_distance, pairwise_distance  # noqa: E402


def _data(kind, rng, n, length):
    if kind == "spike":
        return (np.arange(length)[None, :] == rng.integers(0, length, (n, 1))).astype(float)
    if kind == "runs":
        return np.repeat(rng.random((n, length // 8 + 1)) > 0.5, 8, axis=1)[:, :length].astype(float)
    if kind == "padded":
        return np.cumsum(rng.standard_normal((n, length)), axis=1) * (np.arange(length) < length // 2)
    return (rng.random((n, length)) > 0.5).astype(float)


def _check(monkeypatch, X, Y, metric, r):
    X = torch.as_tensor(X, device="cuda")
    args = (X,) if Y is None else (X, torch.as_tensor(Y, device="cuda"))
    monkeypatch.delenv("WB_GPU_ELASTIC", raising=False)
    got = pairwise_distance(*args, metric=metric, metric_params={"r": r})
    monkeypatch.setenv("WB_GPU_ELASTIC", "ring")
    want = pairwise_distance(*args, metric=metric, metric_params={"r": r})
    np.testing.assert_array_equal(got.cpu().numpy(), want.cpu().numpy())


@pytest.mark.parametrize("metric,r", [("dtw", 0.2), ("dtw", 1.0), ("adtw", 0.4), ("wdtw", 1.0)])
@pytest.mark.parametrize("kind", ["spike", "runs", "padded", "binary"])
@pytest.mark.parametrize("rows,cols", [(20, 6000), (33, 3100), (40, 2500), (500, None)])
def test_shapes(monkeypatch, metric, r, kind, rows, cols):
    rng = np.random.default_rng(rows)
    X = _data(kind, rng, rows, 100)
    Y = None if cols is None else _data(kind, rng, cols, 96)
    _check(monkeypatch, X, Y, metric, r)


@pytest.mark.parametrize("metric,r", [("dtw", 0.2), ("dtw", 1.0), ("adtw", 0.4)])
@pytest.mark.parametrize("rows,cols", [(0, 3), (0, 100), (130, 0), (1, 0), (400, 0), (130, 50)])
def test_some_tied(monkeypatch, metric, r, rows, cols):
    rng = np.random.default_rng(rows + cols)
    X = np.cumsum(rng.standard_normal((700, 100)), axis=1)
    Y = np.cumsum(rng.standard_normal((400, 100)), axis=1)
    X[:rows] = 1.0 + 1e-12 * X[:rows]
    Y[:cols] = 1.0
    _check(monkeypatch, X, Y, metric, r)


@pytest.mark.parametrize("kind", ["spike", "runs"])
def test_argmin(monkeypatch, kind):
    rng = np.random.default_rng(8)
    X, Y = _data(kind, rng, 500, 90), _data(kind, rng, 900, 90)
    kw = dict(k=3, metric="dtw", metric_params={"r": 0.3}, return_distance=True)
    got = argmin_distance(X, Y, **kw)
    monkeypatch.setenv("WB_GPU_ARGMIN", "all")
    for a, b in zip(got, argmin_distance(X, Y, **kw)):
        np.testing.assert_array_equal(a, b)
