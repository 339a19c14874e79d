"""Paired distances whose pairs the guided kernel leaves: none, few (the tail
kernel) and more than that takes (the second pass over their list)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from wildboar_gb300.distance import paired_distance  # noqa: E402


@pytest.mark.parametrize("metric,r", [("dtw", 0.2), ("dtw", 1.0), ("wdtw", 1.0), ("adtw", 0.4)])
@pytest.mark.parametrize("tied", [0, 1, 31, 900, 9001])
def test_same_bits(monkeypatch, metric, r, tied):
    rng = np.random.default_rng(tied)
    X, Y = (np.cumsum(rng.standard_normal((9001, 90)), axis=1) for _ in range(2))
    rows = rng.permutation(9001)[:tied]
    X[rows], Y[rows] = 1.0, (rng.random((tied, 90)) > 0.9).astype(float)
    X, Y = (torch.as_tensor(v, device="cuda") for v in (X, Y))
    monkeypatch.delenv("WB_GPU_ELASTIC", raising=False)
    got = paired_distance(X, Y, metric=metric, metric_params={"r": r})
    monkeypatch.setenv("WB_GPU_ELASTIC", "ring")
    want = paired_distance(X, Y, metric=metric, metric_params={"r": r})
    np.testing.assert_array_equal(got.cpu().numpy(), want.cpu().numpy())
