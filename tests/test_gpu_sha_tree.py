"""SHA-256 trees at the edges of their dispatch, against the oracle: one leaf
up to the one-CTA tree's 128 leaves and past it, rows of 16 bytes (padding in
the same block) up to rows with a padding block of their own.  Hashes are
compared for equality."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lm,r,lb", [(1, 1, 1), (2, 1, 0), (6, 1, 1), (7, 1, 2), (8, 1, 2),
                                     (8, 1, 1), (9, 1, 4), (10, 2, 5), (11, 1, 5), (13, 1, 7)])
def test_sha_tree_equals_oracle(oracle, ctx, lm, r, lb):
    from bitz_gb300 import PcsParams, commit

    msg = oracle.chacha_words(lm * 7 + lb, 1 << lm)
    _, tree, root = oracle.commit(msg, r, lb, 0, n_threads=8)
    c, pd = commit(msg, PcsParams(lm + 7, r, lb, 0), ctx)
    try:
        assert (pd.merkle_tree == tree).all()
        assert c.root == root
    finally:
        pd.free()
