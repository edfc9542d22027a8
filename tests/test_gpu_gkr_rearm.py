"""A proof after one whose transcript paused past a gate arms its rounds again;
after three in a row the context stops.  A gate that runs out costs the launches
of the round that is run again, so the count of launches shows the arming."""
import gc
import time

import pytest
from test_gpu_gkr_armed import _case

pytestmark = pytest.mark.gpu


def test_arming_comes_back_after_a_pause():
    from bitz_gb300 import Context
    from bitz_gb300 import gkr as K
    from oracle import gkr as G

    leaves, zeta = _case()
    own = Context(0)

    class Pausing(G.HashChallenges):
        pause = False

        def challenge(self, stage):
            if self.pause and len(self.messages) == 40:
                time.sleep(0.02)
            return super().challenge(stage)

    def launches(pause):
        tr = Pausing(b"rearm")
        tr.pause = pause
        before = own.kernel_launches()
        K.prove(leaves, 1 << len(zeta), zeta, tr, own)
        return own.kernel_launches() - before

    gc.disable()   # no pause but the test's
    try:
        launches(False)
        plain = launches(False)
        for _ in range(2):   # the second pause meets an armed round again
            assert launches(True) > plain
        assert launches(False) == plain   # and ends the row of proofs with pauses
        for _ in range(3):
            assert launches(True) > plain
        assert launches(True) == plain    # no round is armed any more
    finally:
        gc.enable()
        own.close()
