"""One-CTA SHA-256 trees whose message schedules are computed ahead of the
rounds: fewer leaves than a warp, one to four hashing warps, the shortest rows
that are scheduled ahead and long ones.  Trees and roots equal the oracle's."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lm,r,lb", [(5, 1, 5), (6, 1, 5), (9, 1, 6), (9, 1, 5), (10, 1, 5),
                                     (11, 1, 5), (11, 1, 6), (12, 1, 9), (14, 2, 9)])
def test_tree_equals_oracle(oracle, ctx, lm, r, lb):
    from bitz_gb300 import PcsParams, commit

    msg = oracle.chacha_words(lm * 5 + lb, 1 << lm)
    _, tree, root = oracle.commit(msg, r, lb, 0, n_threads=8)
    for _ in range(3):
        c, pd = commit(msg, PcsParams(lm + 7, r, lb, 0), ctx)
        try:
            assert (pd.merkle_tree == tree).all()
            assert c.root == root
        finally:
            pd.free()
