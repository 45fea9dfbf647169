"""gb_grid_f32_noalloc where its bins are cut into items: one tile that holds
every visibility at and around a multiple of the cut, supports of every
thread-group class, the largest call, a grid with the most bins, and two calls in
a row without a synchronisation between them."""
import numpy as np
import pytest

from tests.test_zz_no_alloc import _case, _geometry, _noalloc, _oracle, _rel

pytestmark = pytest.mark.gpu
TOL32 = 1e-5


@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 1000])
def test_one_dense_tile(n):
    uvw, plane, sup, offs, gcf, vis, G = _case(n, max(n, 100), supports=(8, 13, 40))
    uvw = uvw[:n] * 0.01
    case = (uvw, plane[:n], sup, offs, gcf, vis[:n], G)
    exp = _oracle(case)
    got = _noalloc(case)
    assert np.linalg.norm(got - exp) <= TOL32 * np.linalg.norm(exp)


@pytest.mark.parametrize("n,supports", [(131072, (8, 13, 32)), (131072, (6,)), (60000, (64, 8))])
def test_largest_calls(n, supports):
    case = _case(n + len(supports), n, supports=supports)
    assert _rel(_noalloc(case), _oracle(case)) < TOL32


def test_two_calls_in_a_row_without_a_synchronisation():
    import ctypes as C

    import torch

    from rc_gb300 import lib

    L = lib.load()
    cases = [_case(11, 20000), _case(12, 5000, supports=(16, 8, 40))]
    s = torch.cuda.current_stream().cuda_stream
    held, out = [], []
    for uvw, plane, sup, offs, gcf, vis, G in cases:
        d = [torch.tensor(uvw, device="cuda"), torch.tensor(plane, device="cuda"),
             torch.tensor(vis, dtype=torch.complex64, device="cuda"),
             torch.tensor(gcf, dtype=torch.complex64, device="cuda"),
             torch.zeros((G, G), dtype=torch.complex64, device="cuda"), _geometry(sup, offs, G)]
        held.append(d)
        out.append(d[4])
    torch.cuda.synchronize()
    for d in held:
        lib.check(L.gb_grid_f32_noalloc(C.byref(d[5]), d[2].numel(), d[0].data_ptr(), 3,
                                        d[1].data_ptr(), d[2].data_ptr(), d[3].data_ptr(),
                                        d[4].data_ptr(), s), "gb_grid_f32_noalloc")
    torch.cuda.synchronize()
    for g, c in zip(out, cases):
        assert _rel(g.cpu().numpy(), _oracle(c)) < TOL32
