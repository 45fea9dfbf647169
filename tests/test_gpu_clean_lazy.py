"""The lazy CLEAN loop of gb_hogbom_f32 where it can go wrong, bit for bit
against the numpy float32 loop: more tiles than CTAs, a ragged last tile, a PSF
larger than the image and one smaller than a tile, more components than the
pending list holds, equal peaks, pixels that are not finite, a sparse-coverage
PSF whose sidelobes keep every tile a candidate."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.test_gpu_clean import _run_engine

pytestmark = pytest.mark.gpu


def _psf(rng, pny, pnx, sidelobe):
    p = sidelobe * rng.standard_normal((pny, pnx))
    y, x = np.mgrid[0:pny, 0:pnx]
    p += np.exp(-((y - pny // 2) ** 2 + (x - pnx // 2) ** 2) / 8.0)
    return (p / p[pny // 2, pnx // 2]).astype(np.float32)


def _hogbom_nan(res, psf, ppx, ppy, gain, n_iter):
    """O.hogbom_f32 with a NaN never the peak (numpy's argmax takes the first NaN)."""
    res, model = res.copy(), np.zeros_like(res)
    (ny, nx), (pny, pnx), done = res.shape, psf.shape, 0
    for _ in range(n_iter):
        a = np.where(np.isnan(res), np.float32(-1), np.abs(res))
        py, px = divmod(int(np.argmax(a)), nx)
        if a[py, px] < 0:
            break
        gv = np.float32(gain) * res[py, px]
        s = gv / psf[ppy, ppx]
        dx, dy = px - ppx, py - ppy
        x0, x1, y0, y1 = max(0, dx), min(nx, dx + pnx), max(0, dy), min(ny, dy + pny)
        res[y0:y1, x0:x1] -= s * psf[y0 - dy:y1 - dy, x0 - dx:x1 - dx]
        model[py, px] += gv
        done += 1
    return res, model, done


def _check(res, psf, gain, threshold, n_iter):
    ppy, ppx = psf.shape[0] // 2, psf.shape[1] // 2
    r, m, it = _run_engine(res, psf, ppx, ppy, gain, threshold, n_iter)
    er, em, eit = O.hogbom_f32(res, psf, ppx, ppy, gain, threshold, n_iter)
    assert it == eit
    assert np.array_equal(r, er, equal_nan=True)
    assert np.array_equal(m, em, equal_nan=True)


@pytest.mark.parametrize("ny,nx,pny,pnx,sidelobe,n_iter", [
    (1003, 901, 256, 300, 0.01, 200),  # 240 tiles, ragged
    (200, 333, 700, 801, 0.02, 700),   # PSF past the image, two full lists
    (130, 65, 33, 17, 0.01, 300),      # PSF smaller than a tile
    (64, 64, 64, 64, 0.01, 50),        # one tile
    (1, 5, 3, 3, 0.0, 10),             # less than a tile
    (640, 640, 640, 640, 0.4, 120),    # every tile stays a candidate
])
def test_shapes(ny, nx, pny, pnx, sidelobe, n_iter):
    rng = np.random.default_rng(ny * 7 + nx)
    psf = _psf(rng, pny, pnx, sidelobe)
    res = (0.05 * rng.standard_normal((ny, nx))).astype(np.float32)
    for _ in range(10):
        y, x = rng.integers(0, ny), rng.integers(0, nx)
        res[y, x] += rng.uniform(0.5, 3.0) * rng.choice([-1, 1])
    _check(res, psf, 0.1, 0.0, n_iter)


def test_equal_peaks_in_different_tiles_go_by_the_lowest_index():
    psf = _psf(np.random.default_rng(5), 9, 9, 0.0)
    res = np.zeros((256, 256), np.float32)
    for y, x in [(200, 10), (10, 200), (10, 70), (130, 130)]:
        res[y, x] = -1.5 if x == 70 else 1.5
    _check(res, psf, 0.25, 0.1, 40)
    _check(np.zeros((256, 256), np.float32), psf, 0.25, 0.0, 5)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_pixels_that_are_not_finite(bad):
    rng = np.random.default_rng(6)
    psf = _psf(rng, 200, 200, 0.01)
    res = rng.standard_normal((300, 300)).astype(np.float32)
    res[17, 250] = bad
    for r, p in [(res, psf), (np.full((70, 70), np.nan, np.float32), psf),
                 (np.where(np.isfinite(res), res, 0).astype(np.float32), psf.copy())]:
        if p is not psf:
            p[3, 190] = bad
        got = _run_engine(r, p, 100, 100, 0.1, 0.0, 30)
        with np.errstate(all="ignore"):
            exp = _hogbom_nan(r, p, 100, 100, 0.1, 30)
        assert got[2] == exp[2]
        assert np.array_equal(got[0], exp[0], equal_nan=True)
        assert np.array_equal(got[1], exp[1], equal_nan=True)
