"""When the FP32 dtw forward of few items takes several lanes per item
(wb_dtw32_lanes, host arithmetic): series so long that the lanes' step counts
would leave the int range keep one thread per item."""

import ctypes
import os

import pytest

pytest.importorskip("torch")


def _fn():
    from wildboar_gb300 import _lib
    from wildboar_gb300.distance import batched as B

    if not os.path.exists(_lib.LIB_PATH):
        pytest.skip("libwbgpu.so is not built")
    return _lib.lib().wb_dtw32_lanes, B.Dtw32


def _job(Dtw32, x_len, y_len, r, n_items=2, lengths=False, weighted=False, grid=0):
    j = Dtw32()
    j.x_len, j.y_len, j.nx, j.ny = x_len, y_len, 1, n_items
    j.n_items, j.r, j.grid = n_items, r, grid
    # only whether these are set matters here
    j.x_lengths = j.y_lengths = 8 if lengths else None
    j.weights = 8 if weighted else None
    return j


def _steps(rows, cols, r, strip, lanes):
    """Steps of one item in exact arithmetic."""
    band = max(int(rows * r), 1)
    strips = (rows - 1 + strip - 1) // strip
    reach = min(cols, cols - rows + 2 * band + strip - 2 - lanes * strip)
    delta = max(lanes + 2, reach // 2 + 1)
    return (strips - 1) // lanes * delta + (strips - 1) % lanes + (cols + 1) // 2


@pytest.mark.parametrize("keep", [0, 1])
@pytest.mark.parametrize("lengths", [False, True])
def test_long_series_take_a_thread(keep, lengths):
    fn, Dtw32 = _fn()
    if keep and lengths:
        pytest.skip("kept directions of items with lengths take a thread per item")
    for rows, cols in ((1_000_000, 1_000_000), (910_000, 1_200_000), (500_000, 20_000_000)):
        strip = 16 if keep else 24
        assert _steps(rows, cols, 1.0, strip, 8) * 1 >= 2 ** 31
        assert fn(ctypes.byref(_job(Dtw32, rows, cols, 1.0, lengths=lengths)), keep) == 0
        assert fn(ctypes.byref(_job(Dtw32, cols, rows, 1.0, lengths=lengths)), keep) == 0


@pytest.mark.parametrize("r", [0.001, 0.1, 1.0])
@pytest.mark.parametrize("rows,cols", [(64, 64), (1000, 1000), (3000, 2 ** 27), (200_000, 200_000),
                                       (400_000, 400_000), (10 ** 7, 10 ** 7)])
def test_no_count_leaves_the_int_range(rows, cols, r):
    fn, Dtw32 = _fn()
    for keep in (0, 1):
        strip = fn(ctypes.byref(_job(Dtw32, rows, cols, r)), keep)
        if strip:
            assert max(_steps(rows, cols, r, strip, g) * g * 4 // 32
                       for g in (8, 16, 32)) < 2 ** 30


def test_ordinary_jobs():
    fn, Dtw32 = _fn()
    assert fn(ctypes.byref(_job(Dtw32, 100, 100, 0.1)), 0) == 8
    assert fn(ctypes.byref(_job(Dtw32, 800, 900, 0.1)), 0) == 16
    assert fn(ctypes.byref(_job(Dtw32, 2048, 2048, 0.1, lengths=True)), 0) == 24
    assert fn(ctypes.byref(_job(Dtw32, 200_000, 200_000, 1.0)), 0) == 24
    assert fn(ctypes.byref(_job(Dtw32, 1_000_000, 1_000_000, 1e-4)), 0) == 24
    assert fn(ctypes.byref(_job(Dtw32, 256, 256, 0.2)), 1) == 16
    # one thread per item: weights, an explicit grid, lengths with kept directions
    assert fn(ctypes.byref(_job(Dtw32, 800, 900, 0.1, weighted=True)), 0) == 0
    assert fn(ctypes.byref(_job(Dtw32, 800, 900, 0.1, grid=4)), 0) == 0
    assert fn(ctypes.byref(_job(Dtw32, 256, 256, 0.2, lengths=True)), 1) == 0
    assert fn(ctypes.byref(_job(Dtw32, 0, 9, 0.1)), 0) == -1
    assert fn(None, 0) == -1
