"""Guided FP64 evaluation (32-bit sweep, FP64 on the cells it cannot rule out)
and bit-parallel edr / lcss against the full recurrence: the same bits for every metric it takes,
over its strip and block edges, bands, modes and data that stress its error
bound (ties, constant stretches, near duplicates, offsets, tiny and huge
values)."""

import os

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from wildboar_gb300.distance import paired_distance, pairwise_distance  # noqa: E402

# edr / lcss take the bit-parallel form (full band), whose strips have 32 rows
METRICS = [
    ("edr", {}), ("edr", {"epsilon": 1.0}), ("edr", {"epsilon": 0.3}),
    ("lcss", {}), ("lcss", {"epsilon": 0.4}),
    ("dtw", {"r": 0.1}), ("dtw", {"r": 0.37}), ("dtw", {"r": 1.0}),
    ("ddtw", {"r": 0.3}), ("wdtw", {"r": 1.0}), ("wdtw", {"r": 0.2, "g": 0.3}),
    ("wddtw", {"r": 1.0}), ("adtw", {"r": 0.2}), ("adtw", {"r": 1.0, "p": 0.05}),
    ("adtw", {"r": 0.5, "p": 0.0}),
]
IDS = ["%s-%d" % (m, i) for i, (m, _) in enumerate(METRICS)]
SHAPES = [(1, 5), (33, 1), (31, 33), (32, 32), (64, 64), (65, 65), (57, 130), (131, 60), (256, 249), (25, 400), (400, 26)]


def _full(fn):
    old = os.environ.get("WB_GPU_ELASTIC")
    os.environ["WB_GPU_ELASTIC"] = "ring"
    try:
        return np.asarray(fn())
    finally:
        if old is None:
            os.environ.pop("WB_GPU_ELASTIC", None)
        else:
            os.environ["WB_GPU_ELASTIC"] = old


def _same(fn):
    np.testing.assert_array_equal(np.asarray(fn()), _full(fn))


def _data(kind, rng, n, length):
    w = np.cumsum(rng.standard_normal((n, length)), axis=1)
    if kind == "walk":
        return w
    if kind == "noise":
        return rng.standard_normal((n, length))
    if kind == "integers":  # many exact ties
        return np.round(w)
    if kind == "binary":  # long runs of equal values
        return (w > 0).astype(float)
    if kind == "constant":
        return np.full((n, length), 3.25)
    if kind == "offset":
        return w + 1e9
    if kind == "tiny":
        return w * 1e-200
    if kind == "subnormal":  # whose squares are subnormal
        return w * 1e-160
    if kind == "huge":
        return w * 1e150
    if kind == "outlier":
        w[0, length // 2] = 1e12
        return w
    # near duplicates of one walk
    return w[:1] + 1e-6 * rng.standard_normal((n, length))


@pytest.mark.parametrize("metric,params", METRICS, ids=IDS)
@pytest.mark.parametrize("lx,ly", SHAPES)
def test_pairwise_shapes(metric, params, lx, ly):
    rng = np.random.default_rng(lx * 1009 + ly)
    X, Y = _data("walk", rng, 37, lx), _data("walk", rng, 5, ly)
    _same(lambda: pairwise_distance(X, Y, metric=metric, metric_params=params))


@pytest.mark.parametrize("kind", ["noise", "integers", "binary", "constant", "offset", "tiny",
                                  "subnormal",
                                  "huge", "outlier", "near"])
@pytest.mark.parametrize("metric,params", METRICS, ids=IDS)
def test_pairwise_data(metric, params, kind):
    rng = np.random.default_rng(5)
    X, Y = _data(kind, rng, 34, 150), _data(kind, rng, 6, 150)
    _same(lambda: pairwise_distance(X, Y, metric=metric, metric_params=params))


@pytest.mark.parametrize("metric,params", METRICS, ids=IDS)
def test_singleton_and_paired(metric, params):
    rng = np.random.default_rng(9)
    X, Y = _data("walk", rng, 70, 90), _data("walk", rng, 70, 90)
    _same(lambda: pairwise_distance(X, metric=metric, metric_params=params))
    _same(lambda: paired_distance(X, Y, metric=metric, metric_params=params))


@pytest.mark.parametrize("length,r", [(1100, 1.0), (2048, 0.1), (3000, 0.02)])
def test_long_series(length, r):
    rng = np.random.default_rng(length)
    X, Y = _data("walk", rng, 40, length), _data("walk", rng, 3, length)
    _same(lambda: pairwise_distance(X, Y, metric="dtw", metric_params={"r": r}))
