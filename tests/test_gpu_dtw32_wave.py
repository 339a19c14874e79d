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
