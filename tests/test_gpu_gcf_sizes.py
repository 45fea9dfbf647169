"""gb_gcf_generate over the largest supports of its two routes (no prime factor
above 7: the pruned transforms; others: padded cuFFT) against the oracle's
generator: odd and even supports from one tap to all, both precisions."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("smax", [2, 4, 6, 14, 18, 22, 30, 62, 96, 126, 128, 250])
@pytest.mark.parametrize("tapered", [True, False])
def test_generation_matches_the_oracle(smax, tapered):
    from rc_gb300 import gcf as G

    ws = np.array([-700.0, 0.0, 120.5, 33.0])
    sup = np.array([smax, 1, max(1, smax - 1), max(1, smax // 2)], np.int32)
    tp = 0.2 + np.random.default_rng(smax).uniform(0, 1, smax) if tapered else None
    g64, g32, offs = G.generate(ws, sup, smax, 0.08, taper=tp)
    g64, g32 = g64.cpu().numpy(), g32.cpu().numpy()
    for p, (w, S) in enumerate(zip(ws, sup)):
        exp = O.gcf_layers(w, int(S), smax, 0.08, taper=tp).reshape(-1)
        at = slice(offs[p], offs[p] + 64 * S * S)
        assert rel_l2(g64[at], exp) < 1e-12, (p, w, S)
        assert rel_l2(g32[at], exp) < 1e-6, (p, w, S)
    only32 = G.generate(ws, sup, smax, 0.08, taper=tp, want64=False)[1].cpu().numpy()
    only64 = G.generate(ws, sup, smax, 0.08, taper=tp, want32=False)[0].cpu().numpy()
    assert np.array_equal(only32, g32) and np.array_equal(only64, g64)
