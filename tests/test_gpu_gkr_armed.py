"""GKR rounds enqueued ahead of their challenge: a transcript that takes longer
than the gate waits, or waits on the context's stream itself, gets the same
proof, and one that fails leaves the context usable.  Compared with the
oracle's messages and claim for equality."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case():
    rng = np.random.default_rng(5)
    leaves = rng.integers(0, 2**64, (1 << 12, 2), dtype=np.uint64)
    return leaves, [rng.integers(0, 2**64, 2, dtype=np.uint64) for _ in range(2)]


def _oracle(leaves, zeta):
    from oracle import gkr as G

    _, wit = G.batched_eval(leaves, 1 << len(zeta))
    tr = G.HashChallenges(b"armed")
    point, claim = G.prove(tr.send, tr.challenge, zeta, wit)
    return tr.messages, G.gf_key(claim)


def _prove(ctx, leaves, zeta, act=None):
    from bitz_gb300 import gkr as K
    from oracle import gkr as G

    class Acting(G.HashChallenges):
        def challenge(self, stage):
            if act and len(self.messages) % 17 == 0:
                act()
            return super().challenge(stage)

    tr = Acting(b"armed")
    _, _, claim = K.prove(leaves, 1 << len(zeta), zeta, tr, ctx)
    return tr.messages, G.gf_key(claim)


@pytest.mark.parametrize("how", ["sleep", "synchronize", "fail"])
def test_transcripts_that_hold_the_gate(how):
    from bitz_gb300 import Context

    own = Context(0)
    leaves, zeta = _case()
    exp = _oracle(leaves, zeta)

    def fail():
        raise RuntimeError("no challenge")

    act = {"sleep": lambda: time.sleep(0.02), "synchronize": own.synchronize, "fail": fail}[how]
    try:
        if how == "fail":
            with pytest.raises(RuntimeError):
                _prove(own, leaves, zeta, act)
        else:
            assert _prove(own, leaves, zeta, act) == exp
        assert _prove(own, leaves, zeta) == exp   # the context goes on
    finally:
        own.close()
