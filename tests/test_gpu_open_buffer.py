"""Openings through the context's mapped buffer: the most rows and nodes it
takes and the first that it does not, no nodes, and several threads that open
at once (one holds the buffer, the others take device buffers).  Compared with
the oracle's codeword and multi-proof."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes,q", [(7, 1), (7, 128), (7, 129), (7, 512), (2, 700), (2, 3000),
                                     (0, 64)])
@pytest.mark.parametrize("threads", [1, 4])
def test_rows_and_nodes(oracle, ctx, lanes, q, threads):
    from bitz_gb300 import PcsParams, commit

    log_n, rate, kind = 14, 2, 1
    msg = oracle.chacha_words(q, 1 << log_n)
    cw, tree, _ = oracle.commit(msg, rate, lanes, kind)
    _, pd = commit(msg, PcsParams(log_n + 7, rate, lanes, kind), ctx)
    n_leaves, L = 1 << (log_n - lanes + rate), 1 << lanes
    bad = []

    def one(seed):
        pos = np.sort(np.random.default_rng(seed).choice(n_leaves, q, replace=False))
        rows, proof = pd.rows(pos), pd.multi_proof(pos)
        exp = oracle.merkle_multi_proof(tree, n_leaves, pos.tolist())
        if not ((rows == cw.reshape(n_leaves, L, 2)[pos]).all() and (proof == exp).all()):
            bad.append(seed)

    try:
        ts = [threading.Thread(target=one, args=(i,)) for i in range(threads)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert not bad
    finally:
        pd.free()
