"""Guided evaluation of values that tie everywhere, with more tiles than warps:
the later tiles go to the full recurrence at once, with the same bits."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from wildboar_gb300.distance import pairwise_distance  # noqa: E402


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
