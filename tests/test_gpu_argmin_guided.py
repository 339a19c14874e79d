"""argmin_distance of the dtw family over float32 filters and guided FP64
evaluations: indices (heap order included) and distances bit for bit those of
the all-pairs form (``WB_GPU_ARGMIN=all``), at the filters' tile and chunk
edges and on data that stresses their bounds."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from wildboar_gb300.distance import argmin_distance  # noqa: E402

METRICS = [
    ("dtw", {"r": 0.1}), ("dtw", {"r": 1.0}), ("ddtw", {"r": 0.2}), ("wdtw", {"r": 0.3}),
    ("wddtw", {"r": 1.0, "g": 0.2}), ("adtw", {"r": 0.2, "p": 0.3}), ("adtw", {"r": 1.0}),
]
IDS = ["%s-%d" % (m, i) for i, (m, _) in enumerate(METRICS)]


def _check(monkeypatch, X, Y, **kw):
    got = argmin_distance(X, Y, return_distance=True, **kw)
    monkeypatch.setenv("WB_GPU_ARGMIN", "all")
    want = argmin_distance(X, Y, return_distance=True, **kw)
    monkeypatch.delenv("WB_GPU_ARGMIN")
    for a, b in zip(got, want):
        np.testing.assert_array_equal(np.asarray(a), np.asarray(b))


def _walk(rng, n, length):
    return np.cumsum(rng.standard_normal((n, length)), axis=1)


@pytest.mark.parametrize("metric,params", METRICS, ids=IDS)
@pytest.mark.parametrize("nx,ny,lx,ly,k", [(301, 401, 70, 70, 5), (130, 705, 64, 96, 1),
                                           (517, 163, 101, 60, 10)])
def test_shapes(monkeypatch, metric, params, nx, ny, lx, ly, k):
    rng = np.random.default_rng(nx + ny)
    X, Y = _walk(rng, nx, lx), _walk(rng, ny, ly)
    if lx == ly:  # late near matches and ties
        Y[ny - 3] = X[4] + 1e-3 * rng.standard_normal(lx)
        Y[ny - 2] = Y[ny - 3]
    _check(monkeypatch, X, Y, k=k, metric=metric, metric_params=params)


@pytest.mark.parametrize("kind", ["integers", "constant", "offset", "tiny", "near", "same"])
@pytest.mark.parametrize("metric,params", METRICS, ids=IDS)
def test_data(monkeypatch, metric, params, kind):
    rng = np.random.default_rng(11)
    X, Y = _walk(rng, 300, 66), _walk(rng, 330, 66)
    if kind == "integers":
        X, Y = np.round(X), np.round(Y)
    elif kind == "constant":
        X, Y = np.ones_like(X), np.ones_like(Y)
    elif kind == "offset":
        X, Y = X + 1e8, Y + 1e8
    elif kind == "tiny":
        X, Y = X * 1e-160, Y * 1e-160
    elif kind == "near":
        X, Y = X[:1] + 1e-5 * X, X[:1] + 1e-5 * Y
    else:
        Y[:300] = X
    _check(monkeypatch, X, Y, k=3, metric=metric, metric_params=params)


def test_lower_bound_batches_and_device(monkeypatch):
    rng = np.random.default_rng(3)
    X, Y = _walk(rng, 260, 80), _walk(rng, 400, 80)
    kw = dict(k=4, metric="dtw", metric_params={"r": 0.1})
    lb = np.abs(X[:, None, 0] - Y[None, :, 0])
    _check(monkeypatch, X, Y, lower_bound=lb, **kw)
    monkeypatch.setenv("WB_GPU_ARGMIN_BATCH", str(97 * 400))
    _check(monkeypatch, X, Y, lower_bound=lb, **kw)
    monkeypatch.delenv("WB_GPU_ARGMIN_BATCH")
    Xd, Yd = torch.as_tensor(X, device="cuda"), torch.as_tensor(Y, device="cuda")
    a = argmin_distance(Xd, Yd, return_distance=True, **kw)
    b = argmin_distance(X, Y, return_distance=True, **kw)
    for u, v in zip(a, b):
        np.testing.assert_array_equal(u.cpu().numpy(), v)
