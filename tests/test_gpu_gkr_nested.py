"""A transcript that itself proves on the same context: before a layer's close
(whose entries the last round posts), while a round is armed, and with a pause of
its own behind an armed round of the inner proof.  Both proofs equal the
oracle's."""
import time

import numpy as np
import pytest
from test_gpu_gkr_armed import _case, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("at", [1, 2, 3, 6, 7, 20, 40, 41, 42])
@pytest.mark.parametrize("pause", [False, True])
def test_proof_inside_a_callback(at, pause):
    from bitz_gb300 import Context
    from bitz_gb300 import gkr as K
    from oracle import gkr as G

    own = Context(0)
    leaves, zeta = _case()
    exp = _oracle(leaves, zeta)
    inner = leaves[:256] ^ np.uint64(5)
    exp_inner = _oracle(inner, [])
    got_inner = []

    class Pausing(G.HashChallenges):
        def challenge(self, stage):
            if pause and len(self.messages) == 12:
                time.sleep(0.01)
            return super().challenge(stage)

    class Nested(G.HashChallenges):
        def challenge(self, stage):
            if len(self.messages) == at:
                tr = Pausing(b"armed")
                _, _, claim = K.prove(inner, 1, [], tr, own)
                got_inner.append((tr.messages, G.gf_key(claim)))
            return super().challenge(stage)

    try:
        tr = Nested(b"armed")
        _, _, claim = K.prove(leaves, 1 << len(zeta), zeta, tr, own)
        assert got_inner == [exp_inner]
        assert (tr.messages, G.gf_key(claim)) == exp
    finally:
        own.close()
