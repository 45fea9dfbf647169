"""The engine's FP64 pair where its visibilities are cut into warps' shares: a few,
one per warp, at and above the counts where a share grows, against sums over the
exported index in torch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_sm,extra", [(0, 1), (0, 9), (1, 0), (320, -1), (320, 0), (320, 1), (640, 1)])
def test_pair64_over_the_shares(per_sm, extra):
    import torch

    from rc_gb300.engine import Plan
    from rc_gb300.gcf import layout

    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    rng = np.random.default_rng(n)
    grid, sup = 192, np.array([1, 6, 9], np.int32)
    offs, total = layout(sup)
    uvw = torch.tensor(rng.uniform(-0.52, 0.52, (n, 3)) * grid, device="cuda")
    plane = torch.tensor(rng.integers(-1, len(sup), n).astype(np.int32), device="cuda")
    P = Plan(uvw, scale=1.0, grid_size=grid, grid_shape=(grid, grid), supports=sup, plane=plane)
    gen = torch.Generator(device="cuda").manual_seed(n)
    rand = lambda *shape: torch.randn(*shape, dtype=torch.complex128, device="cuda", generator=gen)
    vis, gcf, model = rand(n), rand(total), rand(grid, grid)
    got = P.grid64(vis, gcf, torch.zeros(grid, grid, dtype=torch.complex128, device="cuda"))
    pred = P.degrid64(gcf, model)
    idx = P.export_index().long()
    ref = torch.zeros(grid * grid, dtype=torch.complex128, device="cuda")
    ref_pred = torch.zeros(n, dtype=torch.complex128, device="cuda")
    for p, s in enumerate(sup.tolist()):
        m = torch.nonzero((idx[:, 4] == 1) & (idx[:, 3] == p))[:, 0]
        k = torch.arange(s * s, device="cuda")
        g = gcf[int(offs[p]) + idx[m, 2][:, None] * s * s + k]
        at = (idx[m, 1][:, None] + k // s) * grid + idx[m, 0][:, None] + k % s
        ref.index_add_(0, at.reshape(-1), (vis[m][:, None] * g).reshape(-1))
        ref_pred[m] = (model.reshape(-1)[at] * g.conj()).sum(1)
    assert bool((idx[:, 4] == 1).any()) or n < 10
    for a, b in ((got.reshape(-1), ref), (pred, ref_pred)):
        assert float(torch.linalg.norm(a - b)) <= 1e-12 * float(torch.linalg.norm(b))
