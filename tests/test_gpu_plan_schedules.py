"""Plans whose commits run side by side take other passes for small codewords
than a commit alone: the largest such codeword, the first larger one, one
commit and one branch, against the oracle's roots and codewords."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,branches", [(1, 4), (3, 1), (5, 4)])
@pytest.mark.parametrize("lm,r,lb", [(15, 2, 6), (16, 2, 5), (17, 1, 4), (17, 2, 7),
                                     (17, 2, 8), (18, 2, 8)])
def test_plan_equals_oracle(oracle, ctx, count, branches, lm, r, lb):
    from bitz_gb300 import BatchPlan, DeviceArray, PcsParams

    msgs = [oracle.chacha_words(100 * lm + i, 1 << lm) for i in range(count)]
    exp = [oracle.commit(m, r, lb, 1, n_threads=8) for m in msgs]
    dev = [DeviceArray.from_host(m, ctx) for m in msgs]
    plan = BatchPlan(dev, [PcsParams(lm + 7, r, lb, 1)] * count, n_branches=branches, ctx=ctx)
    for _ in range(2):
        plan.launch()
        assert [bytes(x) for x in plan.roots()] == [bytes(e[2]) for e in exp]
