"""The FP64 pair over the rules that cut its visibilities into warps' shares (by the
largest support: to 8, to 24, above) and spread gridding's blocks over 512 places of
the visit order: block counts round multiples of 512, shares from the smallest to the
32 that a warp holds and beyond, a core on a few pixels; against sums over the exported
index in torch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(n, supports, share_last=1.0, spread=1.0):
    """share_last: of the visibilities, those of the last (largest) support."""
    import torch

    from rc_gb300.engine import Plan
    from rc_gb300.gcf import layout

    rng = np.random.default_rng(n)
    grid, sup = 128, np.array(supports, np.int32)
    offs, total = layout(sup)
    gen = torch.Generator(device="cuda").manual_seed(n)
    rand = lambda *shape: torch.randn(*shape, dtype=torch.complex128, device="cuda", generator=gen)
    uvw = (torch.rand(n, 3, dtype=torch.float64, device="cuda", generator=gen) - 0.5) * (1.04 * grid * spread)
    plane = rng.integers(-1, max(1, len(sup) - 1), n)
    plane[rng.random(n) < share_last] = len(sup) - 1
    P = Plan(uvw, scale=1.0, grid_size=grid, grid_shape=(grid, grid), supports=sup,
             plane=torch.tensor(plane.astype(np.int32), device="cuda"))
    vis, gcf, model = rand(n), rand(total), rand(grid, grid)
    got = P.grid64(vis, gcf, torch.zeros(grid, grid, dtype=torch.complex128, device="cuda"))
    pred = P.degrid64(gcf, model)
    idx = P.export_index().long()
    ref = torch.zeros(grid * grid, 2, dtype=torch.float64, device="cuda")
    ref_pred = torch.zeros(n, dtype=torch.complex128, device="cuda")
    for p, s in enumerate(sup.tolist()):
        k = torch.arange(s * s, device="cuda")
        for m in torch.nonzero((idx[:, 4] == 1) & (idx[:, 3] == p))[:, 0].split(1 << 17):
            g = gcf[int(offs[p]) + idx[m, 2][:, None] * s * s + k]
            at = (idx[m, 1][:, None] + k // s) * grid + idx[m, 0][:, None] + k % s
            ref.index_add_(0, at.reshape(-1), torch.view_as_real(vis[m][:, None] * g).reshape(-1, 2))
            ref_pred[m] = (model.reshape(-1)[at] * g.conj()).sum(1)
    for a, b in ((got.reshape(-1), torch.view_as_complex(ref)), (pred, ref_pred)):
        assert float(torch.linalg.norm(a - b)) <= 1e-12 * float(torch.linalg.norm(b))


@pytest.mark.parametrize("blocks", [1, 511, 512, 513, 1024, 1025])
@pytest.mark.parametrize("extra", [-1, 0, 1])
def test_blocks_spread_over_the_order(blocks, extra):
    _check(64 * blocks + extra, [3, 8], 0.5)  # eight visibilities a warp, eight warps a block


@pytest.mark.parametrize("supports,per_sm", [([1, 2, 4], 32), ([1, 2, 4], 64), ([1, 9], 80), ([1, 9], 128),
                                             ([1, 25], 320)])
@pytest.mark.parametrize("share,extra", [(1, 0), (1, 1), (8, 1), (31, 1), (32, 0), (32, 1)])
def test_shares(supports, per_sm, share, extra):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    _check(share * per_sm * sms + extra, supports, 0.01)


@pytest.mark.parametrize("n", [40_000, 300_000])
def test_a_dense_core(n):
    _check(n, [4, 8], 0.5, 0.02)
