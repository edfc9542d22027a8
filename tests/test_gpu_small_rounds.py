"""Rounds of few slots: sumcheck folds and messages, and GKR layers, at the
edges of the shared-memory rounds (one CTA, sixteen that each post their sum,
more with a ticket, and the first size of the table kernels).  Compared with
the oracle for equality."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots", [1, 2, 8, 16, 64, 128, 1024, 2048, 4096, 8192, 16384])
@pytest.mark.parametrize("special", [False, True])
def test_folds_and_messages(oracle, ctx, slots, special):
    from bitz_gb300 import DeviceArray
    from bitz_gb300.ligerito import fold_and_msg_lsb, fold_gate_check, round_msg_lsb

    rng = np.random.default_rng(slots)
    n = 4 * slots
    f, b = (rng.integers(0, 2**64, (n, 2), dtype=np.uint64) for _ in range(2))
    r = rng.integers(0, 2**64, 2, dtype=np.uint64)
    if special:
        f[::3] = 2**64 - 1
        b[::2] = 0
        b[1::4] = 2**64 - 1
        r[:] = 2**64 - 1
    df, db = DeviceArray.from_host(f, ctx), DeviceArray.from_host(b, ctx)
    ef, eb, e0, e2 = oracle.fold_and_msg_lsb(f, b, r)
    for nf, nb, (u0, u2) in (fold_and_msg_lsb(df, db, r), fold_gate_check(df, db, r, 0)):
        assert (nf.to_host() == ef).all() and (nb.to_host() == eb).all()
        assert (u0 == e0).all() and (u2 == e2).all()
    m0, m2 = round_msg_lsb(df, db)
    o0, o2 = oracle.round_msg_lsb(f, b)
    assert (m0 == o0).all() and (m2 == o2).all()


@pytest.mark.parametrize("log_n,s", [(2, 0), (5, 1), (9, 0), (13, 3), (16, 0)])
def test_gkr_layers(ctx, log_n, s):
    from bitz_gb300 import gkr as K
    from oracle import gkr as G

    rng = np.random.default_rng(log_n)
    leaves = rng.integers(0, 2**64, (1 << log_n, 2), dtype=np.uint64)
    zeta = [rng.integers(0, 2**64, 2, dtype=np.uint64) for _ in range(s)]
    _, wit = G.batched_eval(leaves, 1 << s)
    exp = G.HashChallenges(b"small")
    _, claim = G.prove(exp.send, exp.challenge, zeta, wit)
    got = G.HashChallenges(b"small")
    _, _, c = K.prove(leaves, 1 << s, zeta, got, ctx)
    assert got.messages == exp.messages and G.gf_key(c) == G.gf_key(claim)
