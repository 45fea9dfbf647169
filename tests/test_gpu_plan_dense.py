"""The plan's work items where one tile holds most of the work: counts at and around
whole items and at the number of them from which a warp takes them together, whole
items between rests of other periods, and the time a plan takes."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plan(n, supports, spread=0.0, grid=256):
    import torch

    from rc_gb300.engine import Plan

    gen = torch.Generator(device="cuda").manual_seed(n)
    uvw = (torch.rand(n, 3, dtype=torch.float64, device="cuda", generator=gen) - 0.5) * (0.8 * grid * spread) + 0.3
    plane = torch.randint(0, len(supports), (n,), dtype=torch.int32, device="cuda", generator=gen)
    make = lambda: Plan(uvw, scale=1.0, grid_size=grid, grid_shape=(grid, grid),
                        supports=np.array(supports, np.int32), plane=plane)
    return make(), make


def _sums(p, supports):
    """The grid's sum for unit visibilities and kernels: every record once."""
    import torch

    n, taps = p.n, sum(int((p.plane_in == k).sum()) * s * s for k, s in enumerate(supports))
    grid = torch.zeros(p.grid_shape, dtype=torch.complex64, device="cuda")
    p.grid(torch.ones(n, dtype=torch.complex64, device="cuda"),
           torch.ones(p.gcf_len, dtype=torch.complex64, device="cuda"), grid)
    return float(grid.real.double().sum()), taps


# tile 24, support 8: an item costs 2 ceil(31^2 / 64) = 32 and 2 a record, and is
# closed at four times 32 (an even share of these counts is less): 48 records
PER = 48


@pytest.mark.parametrize("items", [1, 2, 33, 63, 64, 65, 66, 127, 128, 129, 300])
@pytest.mark.parametrize("extra", [-1, 0, 1])
def test_items_of_one_period(items, extra):
    n = PER * items + extra
    p, _ = _plan(n, [8])
    assert p.stats()["items"] == -(-n // PER) and p.stats()["tiles"] == 1
    got, taps = _sums(p, [8])
    assert got == taps  # whole numbers below 2^24 on every pixel


@pytest.mark.parametrize("n", [500, 5000, 30000])
@pytest.mark.parametrize("supports", [[6, 7, 8], [8, 13, 16, 20, 44], [64, 8]])
def test_items_of_several_periods(n, supports):
    p, _ = _plan(n, supports)
    got, taps = _sums(p, supports)
    assert got == taps


def test_a_dense_tile_costs_no_more_than_spread_ones():
    """4e6 visibilities in one tile against as many over the whole grid: the items'
    kernel aside the dense plan does no more work.  (One thread to the tile: 3 times
    and more.)"""
    import torch

    def best(spread):
        p, make = _plan(4_000_000, [8], spread, 1024)
        p.close()
        t = []
        for _ in range(8):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            q = make()
            t.append(time.perf_counter() - t0)
            q.close()
        return min(t)

    assert best(0.0) < 2.0 * best(1.0)
