"""Results that the device posts to mapped memory: the final polynomial at the
most elements that are posted and the first size that is copied, with
out-of-domain values, and an opening whose proof needs no nodes.  The proofs'
bytes equal the oracle's."""
import pytest

from test_gpu_opening import _prove_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [
    (12, 2, 3, [2], [2, 2], [9, 5], [0, 3], None, [0, 1], 1),   # 128 elements
    (12, 2, 3, [1], [2, 2], [9, 5], [0, 3], None, [0, 2], 1),   # 256
    (8, 1, 4, [4], [1, 1], [32, 2], [0, 0], None, [0, 1], 0),   # 1; every row opened
])
def test_posted_results(oracle, ctx, case):
    _prove_both(oracle, ctx, case, seed=case[3][0] + 7)
