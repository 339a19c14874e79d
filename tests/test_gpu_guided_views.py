"""Guided forms on device arrays that share memory: a set of rows against the
array that it is the start of, and one row against all of it.  The rows after
the shared start are of other sizes than those in it, so a scale taken from the
shared rows alone does not hold for the others."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from wildboar_gb300.distance import argmin_distance, pairwise_distance  # noqa: E402

METRICS = [("dtw", {"r": 0.1}), ("dtw", {"r": 1.0}), ("adtw", {"r": 0.2, "p": 0.3}),
           ("wdtw", {"r": 1.0}), ("ddtw", {"r": 0.2}), ("edr", {"epsilon": 0.7}),
           ("lcss", {"epsilon": 0.7})]
IDS = ["%s-%d" % (m, i) for i, (m, _) in enumerate(METRICS)]


def _walks(times, n=200, length=200, first=1):
    rng = np.random.default_rng(int(times))
    X = np.cumsum(rng.standard_normal((n, length)), axis=1)
    X[first:] *= times * rng.random((n - first, 1))
    return torch.as_tensor(X, device="cuda")


@pytest.mark.parametrize("metric,params", METRICS, ids=IDS)
@pytest.mark.parametrize("times", [2.0, 10.0, 1e6])
@pytest.mark.parametrize("rows", [1, 3, 40])
def test_pairwise(metric, params, times, rows, monkeypatch):
    X = _walks(times, first=rows)
    monkeypatch.delenv("WB_GPU_ELASTIC", raising=False)

    def calls():
        out = [pairwise_distance(X[:rows], X, metric=metric, metric_params=params),
               pairwise_distance(X, X[:rows], metric=metric, metric_params=params)]
        if rows == 1:
            out.append(pairwise_distance(X[0], X, metric=metric, metric_params=params))
        return [np.asarray(o.cpu()) for o in out]

    got = calls()
    monkeypatch.setenv("WB_GPU_ELASTIC", "ring")
    for a, b in zip(got, calls()):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("metric,params", METRICS[:5], ids=IDS[:5])
@pytest.mark.parametrize("rows,batch", [(1, None), (7, None), (200, 60 * 200)])
def test_argmin(metric, params, rows, batch, monkeypatch):
    X = _walks(30.0, first=min(rows, 60))
    if batch:
        monkeypatch.setenv("WB_GPU_ARGMIN_BATCH", str(batch))

    def call():
        return [np.asarray(o.cpu()) for o in
                argmin_distance(X[:rows], X, k=4, metric=metric, metric_params=params,
                                return_distance=True)]

    got = call()
    monkeypatch.setenv("WB_GPU_ARGMIN", "all")
    for a, b in zip(got, call()):
        np.testing.assert_array_equal(a, b)
