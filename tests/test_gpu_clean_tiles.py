"""The lazy CLEAN loop with several tiles to a warp, bit for bit against the numpy
float32 loop: more tiles than a CTA's shared memory holds, several to a lane, equal
peaks in tiles of one warp, the list of components filled; and PSFs of which only a
window can lie on the image, or whose blocks are larger than a tile.  An image one
pixel wide has as many tiles as one 32 times as wide, so most cases are thin."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.test_gpu_clean import _run_engine

pytestmark = pytest.mark.gpu
TILE_W, TILE_H, OWNERS_PER_CTA = 32, 16, 15


def _owners(ny, nx):
    import torch

    tiles = -(-nx // TILE_W) * -(-ny // TILE_H)
    ctas = min(-(-tiles // OWNERS_PER_CTA), torch.cuda.get_device_properties(0).multi_processor_count)
    return tiles, OWNERS_PER_CTA * ctas


def _image(rng, ny, nx, n=40):
    r = (0.05 * rng.standard_normal((ny, nx))).astype(np.float32)
    r[rng.integers(0, ny, n), rng.integers(0, nx, n)] += rng.uniform(-3, 3, n).astype(np.float32)
    return r


def _psf(rng, pny, pnx, ppy, ppx, sidelobe=0.02):
    p = (sidelobe * rng.standard_normal((pny, pnx))).astype(np.float32)
    p[max(0, ppy - 1):ppy + 2, max(0, ppx - 1):ppx + 2] = 0.5
    p[ppy, ppx] = 1
    return p


def _check(res, psf, ppy, ppx, gain, n_iter):
    r, m, it = _run_engine(res, psf, ppx, ppy, gain, 0.0, n_iter)
    er, em, eit = O.hogbom_f32(res, psf, ppx, ppy, gain, 0.0, n_iter)
    assert it == eit
    assert np.array_equal(r, er)
    assert np.array_equal(m, em)


@pytest.mark.parametrize("ny,nx,per_warp,pny,pnx,n_iter", [
    (1501, 2077, 3, 65, 33, 700),           # two tiles and more a warp, a full list
    (600 * 1000, 33, 33, 129, 9, 40),       # two to a lane
    (15_700_000, 1, 431, 257, 3, 25),       # more than shared memory holds
    (700_000, 1, 20, 600_001, 1, 40),       # PSF blocks of 64 pixels
])
def test_several_tiles_to_a_warp(ny, nx, per_warp, pny, pnx, n_iter):
    tiles, owners = _owners(ny, nx)
    assert -(-tiles // owners) >= per_warp or owners > 152 * OWNERS_PER_CTA
    rng = np.random.default_rng(ny + nx)
    _check(_image(rng, ny, nx), _psf(rng, pny, pnx, pny // 2, pnx // 2), pny // 2, pnx // 2, 0.2, n_iter)


def test_equal_peaks_in_tiles_of_one_warp():
    ny, nx = 1_300_000, 1
    tiles, owners = _owners(ny, nx)
    res = np.zeros((ny, nx), np.float32)
    # tiles o, o + owners, .. are a warp's: the second, the last and one of the same lane
    last = (tiles - 1 - 5) // owners
    for k in (0, 1, last, min(32, last)):
        res[(5 + k * owners) * TILE_H + 3, 0] = 1.5 if k % 2 else -1.5
    res[(7 + owners) * TILE_H, 0] = 1.5  # another warp's
    psf = _psf(np.random.default_rng(1), 9, 1, 4, 0, 0.0)
    _check(res, psf, 4, 0, 0.25, 60)


@pytest.mark.parametrize("ny,nx,pny,pnx,ppy,ppx", [
    (64, 64, 1500, 1400, 700, 30),
    (130, 65, 900, 777, 0, 776),
    (20, 300, 4000, 64, 3999, 0),
    (33, 200, 64, 4000, 63, 2000),
    (200, 200, 300, 300, 250, 40),
])
def test_a_window_of_the_psf(ny, nx, pny, pnx, ppy, ppx):
    rng = np.random.default_rng(pny + ppx)
    _check(_image(rng, ny, nx), _psf(rng, pny, pnx, ppy, ppx, 0.2), ppy, ppx, 0.1, 150)
