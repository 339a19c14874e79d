"""Guided evaluation of pairs small against the range of their set, where the
32-bit sweep is coarse and its error bound wide: no cell outside the band may
enter the FP64 recurrence, whose value would then be too small."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from wildboar_gb300.distance import pairwise_distance  # noqa: E402


def _check(monkeypatch, X, Y, metric, params):
    X, Y = (torch.as_tensor(v, device="cuda") for v in (X, Y))
    monkeypatch.delenv("WB_GPU_ELASTIC", raising=False)
    got = pairwise_distance(X, Y, metric=metric, metric_params=params)
    monkeypatch.setenv("WB_GPU_ELASTIC", "ring")
    want = pairwise_distance(X, Y, metric=metric, metric_params=params)
    np.testing.assert_array_equal(got.cpu().numpy(), want.cpu().numpy())


# spikes of four steps of 2^-24 of the range over random levels: some pairs'
# bounds reach the saturated value, which the cells outside the band hold
@pytest.mark.parametrize("seed", [9263, 9440, 9505, 9621, 9935, 10336, 10385, 10893, 11257])
def test_wide_bound(monkeypatch, seed):
    rng = np.random.default_rng(seed)
    length = int(rng.choice([26, 32, 40, 48]))
    r = max(float(rng.choice([0.26, 0.3, 0.35, 0.4, 0.5])), 12.5 / length / 2)
    amplitude = 2.0 ** float(rng.uniform(-25.2, -23.8))
    rate = float(rng.choice([0.03, 0.06, 0.1]))
    X = amplitude * 4 * (rng.random((640, length)) < rate)
    Y = (amplitude * 4 * (rng.random((512, length)) < rate)
         + amplitude * 0.3 * rng.standard_normal((512, 1)))
    X[0, :2] = -1.0, 1.0
    _check(monkeypatch, X, Y, "dtw", {"r": r})


@pytest.mark.parametrize("metric,params", [("dtw", {}), ("adtw", {"p": 0.0}),
                                           ("adtw", {"p": 1e-15})], ids=["dtw", "adtw-0", "adtw"])
@pytest.mark.parametrize("lx,ly,r", [(150, 150, 0.1), (150, 160, 0.08), (400, 400, 0.04),
                                     (64, 64, 0.25)])
@pytest.mark.parametrize("amplitude", [2.0 ** -e for e in (22, 23, 24, 25, 26, 28)])
def test_small_pairs(monkeypatch, metric, params, lx, ly, r, amplitude):
    rng = np.random.default_rng(lx + ly)

    def rows(n, length):
        t, out = np.arange(length), []
        for i in range(n):
            at = rng.integers(0, length)
            out.append([(t > at).astype(float), (np.abs(t - at) < 2).astype(float),
                        np.sin((t + at) / 5.0), rng.standard_normal(length) / 3][i % 4])
        return amplitude * np.array(out)

    X, Y = rows(66, lx), rows(12, ly)
    X[0, :2] = -1.0, 1.0
    _check(monkeypatch, X, Y, metric, {"r": r, **params})
