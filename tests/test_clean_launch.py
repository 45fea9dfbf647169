"""How gb_hogbom_f32 cuts an image for its launch, on a runtime that records the
calls instead of running them: the table of the PSF's block maxima covers what of
the PSF can lie on the image and no more."""
import ctypes as C

import pytest

from tests import fake_runtime

OWNERS = 15  # warps of a CTA that hold tiles
TILE_W, TILE_H, TILE_BYTES = 32, 16, 32
MAX_BLOCKS = 16384


class Args(C.Structure):  # CleanArgs of gb_clean.cu
    _fields_ = [("ptr", C.c_void_p * 4)] + [(k, C.c_int) for k in (
        "nx", "ny", "pnx", "pny", "ppx", "ppy", "ntx", "ntiles", "local")] + [
        ("far", C.c_void_p)] + [(k, C.c_int) for k in (
            "wx0", "wx1", "wy0", "wy1", "eb", "nbx", "nby")] + [
        ("gain", C.c_float), ("threshold", C.c_float), ("n_iter", C.c_int)]


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_runtime.load(str(tmp_path_factory.mktemp("fake")), ["gb_clean"])


def _launch(fake, nx, ny, pnx, pny, ppx, ppy):
    """The arguments and the recorded calls of one call."""
    fake.clear()
    a = Args()
    C.c_void_p.in_dll(fake.lib, "fake_args").value = C.addressof(a)
    C.c_size_t.in_dll(fake.lib, "fake_args_bytes").value = C.sizeof(a)
    n = C.c_int64()
    assert fake.lib.gb_hogbom_work_bytes(nx, ny, C.byref(n)) == 0
    work = C.create_string_buffer(n.value)
    p = C.c_void_p(16)  # never read
    rc = fake.lib.gb_hogbom_f32(p, nx, ny, p, pnx, pny, ppx, ppy, C.c_float(0.1), C.c_float(0.25), 7,
                                p, work, n, None)
    assert rc == 0, fake.ops()
    assert (a.nx, a.ny, a.pnx, a.pny, a.ppx, a.ppy) == (nx, ny, pnx, pny, ppx, ppy)
    assert (a.threshold, a.n_iter) == (0.25, 7)
    return a, fake.ops()


@pytest.mark.parametrize("nx,ny,pnx,pny,ppx,ppy", [
    (64, 64, 4096, 4096, 2048, 2048),
    (65, 130, 777, 900, 776, 0),
    (300, 20, 64, 4000, 0, 3999),
    (2048, 2048, 2048, 2048, 1024, 1024),
    (4200, 4300, 9000, 8000, 4000, 100),
    (1, 1, 3, 3, 1, 1),
])
def test_psf_table_covers_what_can_lie_on_the_image(fake, nx, ny, pnx, pny, ppx, ppy):
    a, _ = _launch(fake, nx, ny, pnx, pny, ppx, ppy)
    for n, pn, pp, w0, w1, nb in ((nx, pnx, ppx, a.wx0, a.wx1, a.nbx), (ny, pny, ppy, a.wy0, a.wy1, a.nby)):
        # a pixel x of the image and a component at c have the PSF's pixel pp + x - c
        assert w0 == max(0, pp - (n - 1)) and w1 == min(pn, pp + n)
        assert (nb - 1 << a.eb) < w1 - w0 <= nb << a.eb
    assert a.nbx * a.nby <= MAX_BLOCKS and a.eb >= 5


@pytest.mark.parametrize("limit", [152, 151, 100, 8, 1])
@pytest.mark.parametrize("nx,ny", [(2048, 2048), (333, 200), (1, 20_000_000)])
def test_fewer_multiprocessors_than_the_device_has(fake, limit, nx, ny):
    """Where a process may use only some of the device's multiprocessors, a
    cooperative launch of one CTA for each of the device's is refused; a smaller one
    runs, and its warps hold all tiles."""
    fake.lib.fake_coop_limit(limit)
    try:
        a, ops = _launch(fake, nx, ny, 9, 9, 4, 4)
    finally:
        fake.lib.fake_coop_limit(1 << 30)
    ran = [o for o in ops if o.startswith("coop")]
    assert len(ran) == 1
    grid, smem = (int(ran[0].split(f"{k}=")[1].split()[0]) for k in ("grid", "smem"))
    assert grid <= limit and (grid * 2 >= limit or grid * OWNERS >= a.ntiles)
    assert a.ntiles == -(-nx // TILE_W) * -(-ny // TILE_H)
    assert a.local * grid * OWNERS >= a.ntiles > (a.local - 1) * grid * OWNERS
    table = -(-a.nbx * a.nby // 4) * 16
    assert smem == table + (0 if a.far else a.local * OWNERS * TILE_BYTES) <= 200 * 1024
    assert bool(a.far) == (table + a.local * OWNERS * TILE_BYTES > 200 * 1024)
