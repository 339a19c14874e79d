"""The lanes-per-item FP32 dtw forward against one thread per item (an explicit
grid), bit for bit."""

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from wildboar_gb300.distance.batched import dtw32  # noqa: E402


# columns up to 100 (strips of 8 rows), 700 (16) and 1700 (24); few and many
# items, a remainder of the items taken together
@pytest.mark.parametrize("high,items", [(9, 3), (40, 1001), (100, 4097), (250, 400), (700, 203),
                                        (1700, 62)])
@pytest.mark.parametrize("r", [0.0, 0.03, 0.2, 1.0])
def test_same_bits_as_one_thread_per_item(high, items, r):
    g = torch.Generator(device="cuda")
    g.manual_seed(high)
    x = torch.randn(items, high, device="cuda", generator=g).cumsum(1)
    y = torch.randn(items, high, device="cuda", generator=g).cumsum(1)
    xl = torch.randint(1, high + 1, (items,), device="cuda", generator=g, dtype=torch.int32)
    yl = torch.randint(1, high + 1, (items,), device="cuda", generator=g, dtype=torch.int32)
    n = items // 4
    xl[:n] = yl[:n]  # equal lengths
    xl[n:n + 4] = torch.tensor([0, 1, 2, high], dtype=torch.int32)[:len(xl[n:n + 4])].cuda()
    t = torch.arange(items, dtype=torch.int32, device="cuda")
    kw = dict(r=r, x_lengths=xl, y_lengths=yl, item_x=t, item_y=t, strip=16, block=64)
    cost = [torch.empty(items, dtype=torch.float64, device="cuda") for _ in range(2)]
    got = dtw32(x, y, out_cost=cost[0], **kw)
    want = dtw32(x, y, out_cost=cost[1], grid=-(-items // 64), **kw)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(got.nan_to_num(-1.0), want.nan_to_num(-1.0))
    assert torch.equal(cost[0].nan_to_num(-1.0), cost[1].nan_to_num(-1.0))


@pytest.mark.parametrize("nx,ny,lx,ly", [(7, 5, 33, 64), (20, 9, 300, 129), (3, 4, 1600, 1700)])
def test_grid_items(nx, ny, lx, ly):
    g = torch.Generator(device="cuda")
    g.manual_seed(nx)
    x = torch.randn(nx, lx, device="cuda", generator=g)
    y = torch.randn(ny, ly, device="cuda", generator=g)
    assert torch.equal(dtw32(x, y, r=0.1), dtw32(x, y, r=0.1, grid=2))


@pytest.mark.parametrize("nx,ny,lx,ly,r", [(1, 1, 1, 5, 0.1), (3, 2, 16, 17, 0.0), (5, 7, 33, 64, 0.3),
                                           (70, 3, 257, 129, 0.1), (40, 2, 600, 600, 1.0)])
def test_kept_directions(nx, ny, lx, ly, r):
    """The kept sweep of few items and its walk against one thread per item."""
    import ctypes

    from wildboar_gb300 import _lib
    from wildboar_gb300.distance import batched as B

    g = torch.Generator(device="cuda")
    g.manual_seed(lx)
    x = torch.randn(nx, lx, device="cuda", generator=g).cumsum(1)
    y = torch.randn(ny, ly, device="cuda", generator=g).cumsum(1)
    up = torch.rand(nx * ny, device="cuda", generator=g, dtype=torch.float64)
    res = []
    for grid in (0, 3):
        job = B.make_job(x, y, r=r, grid=grid)
        keep = torch.zeros(_lib.lib().wb_dtw32_keep_bytes(ctypes.byref(job)), dtype=torch.uint8,
                           device="cuda")
        out = torch.empty(nx * ny, dtype=torch.float64, device="cuda")
        _lib.check(_lib.lib().wb_dtw32_distance_keep(ctypes.byref(job), out.data_ptr(), None,
                                                     keep.data_ptr(), keep.numel(), B._stream()))
        gx, gy = torch.zeros_like(x), torch.zeros_like(y)
        _lib.check(_lib.lib().wb_dtw32_backward_keep(
            ctypes.byref(job), out.data_ptr(), up.data_ptr(), gx.data_ptr(), lx, gy.data_ptr(),
            ly, keep.data_ptr(), keep.numel(), B._stream()))
        res.append((out, keep, gx, gy))
    (out, keep, gx, gy), (out1, keep1, gx1, gy1) = res
    assert torch.equal(out, out1)
    # the direction words of whole strips (rows past the series' end carry no
    # direction, and groups of 8 words are written whole)
    n, m = min(lx, ly), max(lx, ly)
    w = max(int(n * r), 1)
    words = sum(min(m, 16 * s + 16 + m - n + w) - max(0, 2 + 16 * s - w)
                for s in range((n - 1) // 16))
    strips = max((n + 14) // 16, 1)
    table = -(-2 * strips * 4 // 256) * 64
    at = torch.arange(words, device="cuda")
    for kept in (keep.view(torch.int32), keep1.view(torch.int32)):
        batches = kept.view(-(-nx * ny // 32), -1)
        lanes = batches[:, table:].reshape(batches.shape[0], -1, 32, 8).transpose(1, 2)
        lanes = lanes.reshape(batches.shape[0] * 32, -1)[:nx * ny, at]
        res.append((lanes, batches[:, :strips], batches[:, strips:2 * strips]))
    for a, b in zip(res[2], res[3]):
        assert torch.equal(a, b)
    # sums over the other side's series, added in any order
    torch.testing.assert_close(gx, gx1, rtol=2e-5, atol=2e-5)
    torch.testing.assert_close(gy, gy1, rtol=2e-5, atol=2e-5)
