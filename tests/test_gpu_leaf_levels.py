"""BLAKE3 trees whose lower levels the leaf kernel builds, at the edges of that
rule (one launch saved or not, short leaves and leaves of one to sixteen
chunks), and the roots of synchronous commits, which the last kernel posts,
against the oracle; hashes are compared for equality."""
import pytest

pytestmark = pytest.mark.gpu


# (log_msg_len, log_inv_rate, log_batch_size): 2^9 .. 2^18 leaves
@pytest.mark.parametrize("lm,r,lb", [(11, 1, 1), (12, 1, 2), (12, 1, 1), (13, 1, 0), (17, 1, 1),
                                     (14, 1, 6), (15, 1, 6), (16, 1, 6), (15, 1, 7), (17, 1, 8),
                                     (18, 1, 9), (18, 2, 10), (20, 1, 6), (17, 1, 0)])
def test_tree_equals_oracle(oracle, ctx, lm, r, lb):
    from bitz_gb300 import PcsParams, commit

    msg = oracle.chacha_words(lm * 5 + lb, 1 << lm)
    _, tree, root = oracle.commit(msg, r, lb, 1, n_threads=8)
    c, pd = commit(msg, PcsParams(lm + 7, r, lb, 1), ctx)
    try:
        assert (pd.merkle_tree == tree).all()
        assert c.root == root
    finally:
        pd.free()


def test_more_commits_than_root_slots(oracle, ctx):
    """Roots of commits kept open past the mailbox's slots stay their own."""
    from bitz_gb300 import PcsParams, commit

    kept = []
    for i in range(40):
        lm = 6 + i % 5
        msg = oracle.chacha_words(900 + i, 1 << lm)
        kept.append((commit(msg, PcsParams(lm + 7, 1, 2, i % 2), ctx),
                     oracle.commit(msg, 1, 2, i % 2, n_threads=2)[2]))
    for (c, pd), root in kept:
        assert c.root == root
        assert pd.merkle_tree[-1].tobytes() == root
        pd.free()
