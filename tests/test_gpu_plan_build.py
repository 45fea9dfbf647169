"""The plan's tables where their kernels can go wrong: bin counts at and around
the scan's block size and far above it, one bin with every visibility (many items
of one tile), bins with one each, cut footprints, nothing kept, no visibilities.
The FP32 pair on them against the plain FP64 pair, and the counts against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,grid,tile,supports,spread", [
    (0, 256, 24, (8,), 1.0),
    (1, 256, 24, (8, 12), 1.0),
    (5000, 512, 8, (8,), 1.0),         # 64 x 64 tiles: 4096 bins
    (5000, 504, 8, (9,), 1.0),         # 3969
    (5000, 520, 8, (8,), 1.0),         # 4225
    (3000, 4096, 8, (8, 15, 44), 1.0),  # 262144 tiles of three periods
    (200000, 256, 24, (8, 20, 44), 0.0),  # one place
    (50000, 256, 32, (6, 13, 70), 0.05),
    (2000, 128, 24, (40,), 30.0),      # mostly out of bounds
    (300, 96, 24, (90,), 50.0),        # nothing kept
])
def test_pair_on_the_plans_tables(n, grid, tile, supports, spread):
    import torch

    from rc_gb300.engine import Plan
    from rc_gb300.gcf import layout

    rng = np.random.default_rng(n + grid + tile)
    sup = np.array(supports, np.int32)
    offs, total = layout(sup)
    uv = rng.uniform(-0.4, 0.4, (n, 2)) * grid * spread + 0.3
    uvw = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
    uvw[:, :2] = torch.tensor(uv, device="cuda")
    plane = rng.integers(-1, len(sup), n).astype(np.int32)
    P = Plan(uvw, scale=1.0, grid_size=grid, grid_shape=(grid, grid), supports=sup,
             plane=torch.tensor(plane, device="cuda"), tile=tile)
    idx = P.export_index().cpu().numpy() if n else np.zeros((0, 5), np.int32)
    keep = idx[:, 4] == 1
    s2 = sup.astype(np.int64)[np.maximum(idx[:, 3], 0)] ** 2
    st = P.stats()
    assert st["kept"] == keep.sum() and st["taps"] == s2[keep].sum()
    cell = set(zip(idx[keep, 0] // tile, idx[keep, 1] // tile))
    assert st["tiles"] >= len(cell) and (st["items"] > 0) == bool(keep.any())
    gen = torch.Generator(device="cuda").manual_seed(n)
    rand = lambda *shape: torch.randn(*shape, dtype=torch.complex128, device="cuda", generator=gen)
    vis, gcf, model = rand(n), rand(total), rand(grid, grid)
    g64 = torch.zeros(grid, grid, dtype=torch.complex128, device="cuda")
    g32 = torch.zeros(grid, grid, dtype=torch.complex64, device="cuda")
    P.grid64(vis, gcf, g64)
    P.grid(vis.to(torch.complex64), gcf.to(torch.complex64), g32)
    p32 = P.degrid(gcf.to(torch.complex64), model.to(torch.complex64))
    p64 = P.degrid64(gcf, model)
    for a, b in ((g32, g64), (p32, p64)):
        assert float(torch.linalg.norm(a - b)) <= 1e-5 * float(torch.linalg.norm(b))
    # every visibility once in the visit order: the FP64 pair reads it, so a
    # second run on a permutation of the input gives the same grid
    if n > 1:
        perm = torch.randperm(n, device="cuda", generator=gen)
        Q = Plan(uvw[perm].contiguous(), scale=1.0, grid_size=grid, grid_shape=(grid, grid),
                 supports=sup, plane=torch.tensor(plane, device="cuda")[perm].contiguous(), tile=tile)
        h64 = torch.zeros_like(g64)
        Q.grid64(vis[perm].contiguous(), gcf, h64)
        assert float(torch.linalg.norm(h64 - g64)) <= 1e-12 * float(torch.linalg.norm(g64))
