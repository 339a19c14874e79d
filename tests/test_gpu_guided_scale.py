"""Guided evaluation of pairs far smaller than the range of their set, whose
scale in 32 bits is at its end: adtw with penalties from 0 up, wdtw with weights
down to 0, against the full recurrence bit for bit."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from wildboar_gb300.distance import argmin_distance, pairwise_distance  # noqa: E402


def _sets(amplitude, lx, ly):
    """Values in [-1, 1], symmetric about 0, half of the series of `amplitude`
    (steps of it, one series the other shifted)."""
    rng = np.random.default_rng(lx + ly)

    def one(n, length):
        A = rng.uniform(-1.0, 1.0, (n, length))
        A[0, 0], A[0, 1] = -1.0, 1.0
        for i in range(1, n, 2):
            step = (np.arange(length) > length // 3 + i).astype(float)
            A[i] = amplitude * (step + np.round(3 * rng.standard_normal(length)) / 4)
        A[n - 1] = amplitude * np.roll(A[1] / amplitude, 1)
        return A

    return one(34, lx), one(9, ly)


def _check(monkeypatch, X, Y, metric, params):
    monkeypatch.delenv("WB_GPU_ELASTIC", raising=False)
    got = pairwise_distance(X, Y, metric=metric, metric_params=params)
    monkeypatch.setenv("WB_GPU_ELASTIC", "ring")
    np.testing.assert_array_equal(
        got, pairwise_distance(X, Y, metric=metric, metric_params=params))


@pytest.mark.parametrize("amplitude", [1e-6, 1e-12, 1e-14, 1e-16, 1e-17, 1e-18, 1e-30])
@pytest.mark.parametrize("lx,ly", [(60, 60), (60, 90), (150, 150)])
@pytest.mark.parametrize("r", [0.3, 1.0])
@pytest.mark.parametrize("p", [0.0, 1e-300, 1e-40, 1e-33, 1e-20, 1.0])
def test_adtw(monkeypatch, amplitude, lx, ly, r, p):
    _check(monkeypatch, *_sets(amplitude, lx, ly), "adtw", {"r": r, "p": p})


@pytest.mark.parametrize("amplitude", [1e-6, 1e-16, 1e-18])
@pytest.mark.parametrize("lx,ly", [(60, 60), (60, 90)])
def test_dtw(monkeypatch, amplitude, lx, ly):
    _check(monkeypatch, *_sets(amplitude, lx, ly), "dtw", {"r": 0.3})


# g n / 2 of 60 to 800: weights near the main diagonal of e^-60 down to 0
@pytest.mark.parametrize("g", [0.4, 0.6, 0.8, 1.0, 1.5, 2.5, 8.0, np.inf])
@pytest.mark.parametrize("lx,ly", [(200, 200), (200, 180), (150, 200)])
@pytest.mark.parametrize("r", [0.3, 1.0])
@pytest.mark.parametrize("times", [1.0, 1e-17, 1e200])
def test_wdtw(monkeypatch, g, lx, ly, r, times):
    rng = np.random.default_rng(lx)
    X = times * np.cumsum(rng.standard_normal((34, lx)), axis=1)
    Y = times * np.cumsum(rng.standard_normal((5, ly)), axis=1)
    X[3:9, ::7] *= -1.0
    _check(monkeypatch, X, Y, "wdtw", {"r": r, "g": g})


@pytest.mark.parametrize("g", [0.8, 2.5, np.inf])
def test_wdtw_argmin(monkeypatch, g):
    rng = np.random.default_rng(7)
    X = np.cumsum(rng.standard_normal((70, 200)), axis=1)
    Y = np.cumsum(rng.standard_normal((300, 200)), axis=1)
    kw = dict(k=3, metric="wdtw", metric_params={"r": 0.5, "g": g}, return_distance=True)
    got = argmin_distance(X, Y, **kw)
    monkeypatch.setenv("WB_GPU_ARGMIN", "all")
    for a, b in zip(got, argmin_distance(X, Y, **kw)):
        np.testing.assert_array_equal(a, b)


# penalties just above a float: each move is off by up to 2^-23 of it
@pytest.mark.parametrize("length", [25, 28, 60, 300])
@pytest.mark.parametrize("moves", [2, 8, 40])
def test_adtw_penalty_rounding(monkeypatch, length, moves):
    rng = np.random.default_rng(length)
    X = rng.integers(-512, 513, (64, length)) / 512.0
    Y = np.roll(X[:12], 2, axis=1)
    X[0, 0], X[0, 1] = -1.0, 1.0
    p = (1.0 + 2.0 ** -23 + 2.0 ** -40) * length / (8.0 * moves)
    _check(monkeypatch, X, Y, "adtw", {"r": 0.5, "p": p})
