"""The reference-ABI pair where a call's records are cut into chunks and warps'
shares: one record, counts at and above those where a share grows, sparse edges
round a dense core, nothing kept, against the oracle (FP64, relative L2 1e-12)."""
import numpy as np
import pytest

from oracle import oracle as O
from rc_gb300 import compat
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,per_sm,extra", [(8, 0, 1), (8, 128, 1), (16, 0, 3), (16, 20, 1), (16, 128, 0),
                                            (16, 256, 1), (32, 32, 1), (64, 2, 1)])
@pytest.mark.parametrize("spread", [0.15, 50.0])
def test_abi_pair_over_the_shares(S, per_sm, extra, spread):
    import torch

    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    rng = np.random.default_rng(n + S)
    G = 320
    vis5 = np.zeros((n, 5))
    vis5[:, :2] = rng.standard_normal((n, 2)) * spread * G
    vis5[0, :2] = 2.5 if spread < 1 else 1e9
    vis5[:, 3:] = rng.standard_normal((n, 2))
    gcf = rng.standard_normal((64, S, S)) + 1j * rng.standard_normal((64, S, S))
    got, exp = np.zeros((G, G), np.complex128), np.zeros((G, G), np.complex128)
    assert compat.call_scatter("kern_scatter_gpu1", 1.0, G, 64, vis5, gcf, got) == 0
    O.scatter(1.0, G, 64, vis5, gcf, exp)
    assert np.abs(exp).sum() > 0 or spread > 1
    assert np.linalg.norm(got - exp) <= 1e-12 * np.linalg.norm(exp)
    model = rng.standard_normal((G, G)) + 1j * rng.standard_normal((G, G))
    out = np.zeros_like(vis5)
    assert compat.call_degrid("kern_degrid_gpu1", 1.0, G, 64, gcf, model, vis5, out) == 0
    assert rel_l2(out[:, 3:], O.degrid(1.0, G, 64, gcf, model, vis5)[:, 3:]) < 1e-12
