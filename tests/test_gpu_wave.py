"""erp, msm and twe over the full band: strips of a pair over the lanes of a
warp against the one-thread-per-pair ring kernel, bit for bit."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from wildboar_gb300.distance import paired_distance, pairwise_distance  # noqa: E402

METRICS = [
    ("erp", {"g": 0.0}),
    ("erp", {"g": 0.7}),
    ("msm", {"c": 1.0}),
    ("msm", {"c": 0.0}),
    ("msm", {"c": 1e-9}),
    ("twe", {"penalty": 1.0, "stiffness": 0.001}),
    ("twe", {"penalty": 0.25, "stiffness": 0.5}),
]
# strips of 8 rows on 1 to 32 lanes: whole strips and remainders, fewer columns
# than lanes, more strips than lanes, one pair and many
SIZES = [(1, 1, 2, 2), (1, 1, 9, 3), (3, 2, 8, 8), (3, 2, 17, 33), (2, 2, 257, 40),
         (2, 3, 300, 31), (5, 7, 64, 65), (40, 31, 100, 90), (61, 47, 33, 257),
         (150, 130, 24, 24), (401, 395, 26, 31)]


def _data(kind, n, length, rng):
    a = rng.standard_normal((n, length))
    if kind == "walk":
        return np.cumsum(a, axis=1)
    if kind == "grid":  # ties everywhere
        return np.round(a * 2) / 2
    return a * 10.0 ** rng.integers(-12, 13, size=(n, length))


@pytest.mark.parametrize("metric,params", METRICS)
@pytest.mark.parametrize("kind", ["walk", "grid", "wide"])
def test_same_bits_as_the_ring_kernel(metric, params, kind, monkeypatch):
    rng = np.random.default_rng(len(kind))
    for nx, ny, lx, ly in SIZES:
        X, Y = _data(kind, nx, lx, rng), _data(kind, ny, ly, rng)

        def calls():
            k = min(nx, ny)
            out = [pairwise_distance(X, Y, metric=metric, metric_params=params)]
            if nx > 1:
                out.append(pairwise_distance(X, metric=metric, metric_params=params))
            if lx == ly:
                out.append(paired_distance(X[:k], Y[:k], metric=metric, metric_params=params))
            return out

        monkeypatch.delenv("WB_GPU_ELASTIC", raising=False)
        got = calls()
        monkeypatch.setenv("WB_GPU_ELASTIC", "ring")
        for a, b in zip(got, calls()):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("metric", ["erp", "msm", "twe"])
def test_dims_and_device_inputs(metric, monkeypatch):
    """A dim of a multivariate set (strided rows), host and device, float32 and
    a reversed view."""
    rng = np.random.default_rng(3)
    X = np.cumsum(rng.standard_normal((9, 3, 41)), axis=2)
    Y = np.cumsum(rng.standard_normal((6, 3, 50)), axis=2)

    def calls():
        xd, yd = torch.as_tensor(X, device="cuda"), torch.as_tensor(Y, device="cuda")
        return [
            pairwise_distance(X, Y, dim=2, metric=metric),
            pairwise_distance(X, dim=1, metric=metric),
            pairwise_distance(xd, yd, dim=1, metric=metric).cpu().numpy(),
            pairwise_distance(X[::-1, :, ::-1], Y, dim=0, metric=metric),
            pairwise_distance(X.astype(np.float32), Y.astype(np.float32), dim=0, metric=metric),
        ]

    monkeypatch.delenv("WB_GPU_ELASTIC", raising=False)
    got = calls()
    monkeypatch.setenv("WB_GPU_ELASTIC", "ring")
    for a, b in zip(got, calls()):
        np.testing.assert_array_equal(a, b)
