"""erp, msm and twe over the full band with pairs enough for one lane each: last
strips of every number of rows, and twe on both sides of the rule that leaves many
short series to the ring kernel.  Bit for bit the ring kernel."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from wildboar_gb300.distance import pairwise_distance  # noqa: E402


def _walk(n, length, seed):
    rng = np.random.default_rng(seed)
    return torch.as_tensor(np.cumsum(rng.standard_normal((n, length)), axis=1), device="cuda")


@pytest.mark.parametrize("metric", ["erp", "msm", "twe"])
@pytest.mark.parametrize("lx", [2, 8, 9, 24, 25, 26, 27, 28, 29, 30, 31, 33])
@pytest.mark.parametrize("nx,ny", [(601, 800), (96, 5000), (80, 5000)])
def test_same_bits(monkeypatch, metric, lx, nx, ny):
    X, Y = _walk(nx, lx, lx), _walk(ny, 29, 1)
    monkeypatch.delenv("WB_GPU_ELASTIC", raising=False)
    got = pairwise_distance(X, Y, metric=metric)
    monkeypatch.setenv("WB_GPU_ELASTIC", "ring")
    np.testing.assert_array_equal(got.cpu().numpy(),
                                  pairwise_distance(X, Y, metric=metric).cpu().numpy())
