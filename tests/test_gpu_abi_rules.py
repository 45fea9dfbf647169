"""The reference-ABI pair at the counts where its rules change: four small records to
a warp from where every multiprocessor has eight warps, and the 32 that a warp holds at
most (the cases of tests/test_gpu_abi_shares.py at other counts)."""
import pytest

from tests.test_gpu_abi_shares import test_abi_pair_over_the_shares as _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,per_sm,extra", [(S, p, e) for S in (8, 16) for p in (8, 16, 32) for e in (-1, 0, 1)] +
                         [(32, 8, 1), (8, 32 * 128, 0), (8, 32 * 128, 1)])
def test_pair_where_a_share_grows(S, per_sm, extra):
    _pair(S, per_sm, extra, 0.15)
