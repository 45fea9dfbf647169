"""gb_grid_f32_noalloc with more (class, tile) bins than its one-block scan has
threads: several bins to a thread, class boundaries inside a thread's share, and as
many bins as a call may have; against the oracle.  Captured in a graph.  And on the
bounds-checked build, where a record index must lie below this call's own number of
records, after a call with more of them."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from tests.test_zz_no_alloc import _case, _geometry, _noalloc, _oracle, _rel

pytestmark = pytest.mark.gpu
TOL32 = 1e-5
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("G,supports", [
    (1024, (8,)),            # 32 x 32 tiles: a bin to a thread
    (1030, (8, 9)),          # 33 x 33: two to a thread
    (2000, (8, 13, 32)),     # three classes, boundaries inside a share
    (4096, (6, 16, 24, 64)),  # four
    (8192, (8,)),            # 65,536 bins, the most
])
def test_many_bins(G, supports):
    from rc_gb300 import lib

    n = 20000
    assert (-(-G // 32)) ** 2 <= lib.NOALLOC_MAX_BINS
    case = _case(G + len(supports), n, G=G, supports=supports)
    assert _rel(_noalloc(case), _oracle(case)) < TOL32


def test_one_bin_too_many_is_refused():
    from rc_gb300 import lib

    with pytest.raises(lib.GbError) as e:
        _noalloc(_case(3, 100, G=8193, supports=(8,)))
    assert e.value.code == lib.ERR_CAPACITY


def test_in_a_cuda_graph():
    import ctypes as C

    import torch

    from rc_gb300 import lib

    L = lib.load()
    case = _case(21, 9000, G=1000, supports=(8, 20, 40))
    uvw, plane, sup, offs, gcf, vis, G = case
    d = [torch.tensor(uvw, device="cuda"), torch.tensor(plane, device="cuda"),
         torch.tensor(vis, dtype=torch.complex64, device="cuda"),
         torch.tensor(gcf, dtype=torch.complex64, device="cuda")]
    out, geo = torch.zeros((G, G), dtype=torch.complex64, device="cuda"), _geometry(sup, offs, G)
    torch.cuda.synchronize()
    s, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        lib.check(L.gb_grid_f32_noalloc(C.byref(geo), len(vis), d[0].data_ptr(), 3, d[1].data_ptr(),
                                        d[2].data_ptr(), d[3].data_ptr(), out.data_ptr(),
                                        s.cuda_stream), "gb_grid_f32_noalloc")
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert _rel(out.cpu().numpy(), _oracle(case)) < TOL32


_CHILD = r"""
import ctypes as C, json, sys
sys.path.insert(0, sys.argv[1])
from rc_gb300 import lib
from tests.test_zz_no_alloc import _case, _noalloc, _oracle, _rel
L = lib.load()
v = C.c_int64()
L.gb_checked_violations(C.byref(v))
out = {"library": L._name, "rel": []}
for n, sup in ((131072, (8, 13)), (3, (8,)), (500, (8, 40)), (20000, (64, 8)), (1, (16,))):
    c = _case(n, max(n, 100), supports=sup)
    c = (c[0][:n] * 0.3,) + (c[1][:n],) + c[2:5] + (c[5][:n], c[6])
    e = _oracle(c)
    out["rel"].append(float(abs(_noalloc(c) - e).max() / max(abs(e).max(), 1e-30)))
L.gb_checked_violations(C.byref(v))
out["violations"] = v.value
print(json.dumps(out))
"""


def test_checked_build_bounds_records_by_this_call():
    from rc_gb300 import build as B

    lib_path = B.build(checked=True)
    env = dict(os.environ, RC_GB300_CHECKED="1", RC_GB300_AUTOBUILD="0")
    r = subprocess.run([sys.executable, "-c", _CHILD, ROOT], env=env, capture_output=True, text=True,
                       timeout=1500)
    assert r.returncode == 0, r.stderr[-4000:]
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert os.path.samefile(out["library"], lib_path)
    assert max(out["rel"]) < 1e-4 and out["violations"] == 0
