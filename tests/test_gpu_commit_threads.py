"""More threads than the mailbox has slots for roots commit on one context at
once: every commit returns its own root, the oracle's."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def test_more_threads_than_root_slots(oracle, ctx):
    from bitz_gb300 import DeviceArray, PcsParams, commit

    cases = []
    for i in range(48):
        lm = 6 + i % 5
        msg = oracle.chacha_words(700 + i, 1 << lm)
        cases.append((DeviceArray.from_host(msg, ctx), PcsParams(lm + 7, 1, 2, i % 2),
                      oracle.commit(msg, 1, 2, i % 2, n_threads=2)[2]))
    for d, p, _ in cases:   # twiddles and kernels of every shape are loaded
        commit(d, p, ctx)[1].free()
    wrong, start = [], threading.Barrier(len(cases))

    def work(d, p, root):
        start.wait()
        for _ in range(40):
            try:
                c, pd = commit(d, p, ctx)
                if c.root != root:
                    wrong.append((p, "root"))
                pd.free()
            except Exception as e:
                wrong.append((p, e))

    threads = [threading.Thread(target=work, args=c) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, (len(wrong), wrong[:3])
