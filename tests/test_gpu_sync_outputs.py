"""What a synchronous call leaves on the device, read at once on another
non-blocking stream: the tree and codeword of a commit, whose root the last
kernel posts (one-CTA trees of both hashes, levels above leaf kernels), and the
folded arrays of a public fold, whose message one to sixteen CTAs or the last of
many post; and the leaves buffer that a grand-product proof folds in.  Compared
with the oracle for equality."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def other():
    """A second context: its stream reads what the first one's calls wrote."""
    from bitz_gb300 import Context

    c = Context(0)
    yield c
    c.close()


def _read(other, ptr, shape, dtype):
    from bitz_gb300 import _lib, lib

    a = np.zeros(shape, dtype)
    assert lib().bz_memcpy_d2h(other.handle, _lib.ptr(a), ctypes.c_void_p(ptr), a.nbytes) == 0
    return a


# (log_msg_len, log_inv_rate, log_batch_size, hash)
@pytest.mark.parametrize("lm,r,lb,h", [(8, 1, 3, 1), (10, 1, 5, 0), (12, 1, 2, 1), (14, 2, 7, 1),
                                       (14, 1, 2, 0), (17, 1, 1, 1)])
def test_tree_on_another_stream(oracle, ctx, other, lm, r, lb, h):
    from bitz_gb300 import DeviceArray, PcsParams, commit

    msg = oracle.chacha_words(lm + 31 * lb, 1 << lm)
    cw, tree, root = oracle.commit(msg, r, lb, h, n_threads=8)
    d_msg = DeviceArray.from_host(msg, ctx)
    for i in range(32):
        c, pd = commit(d_msg, PcsParams(lm + 7, r, lb, h), ctx)
        p_cw, p_tree = pd.device_ptrs()
        got = _read(other, p_tree, tree.shape, np.uint8)
        assert c.root == root
        assert (got == tree).all()
        if i == 0:
            assert (_read(other, p_cw, cw.shape, np.uint64) == cw).all()
        pd.free()


@pytest.mark.parametrize("log_n", [1, 2, 4, 8, 10, 14, 15, 16, 18])
def test_folds_on_another_stream(oracle, ctx, other, log_n):
    from bitz_gb300 import DeviceArray
    from bitz_gb300.ligerito import fold_and_msg_lsb

    rng = np.random.default_rng(log_n)
    n = 1 << log_n
    f, b = (rng.integers(0, 2**64, (n, 2), dtype=np.uint64) for _ in range(2))
    r = rng.integers(0, 2**64, 2, dtype=np.uint64)
    ef, eb, e0, e2 = oracle.fold_and_msg_lsb(f, b, r)
    d_f, d_b = DeviceArray.from_host(f, ctx), DeviceArray.from_host(b, ctx)
    for _ in range(32):
        nf, nb, (u0, u2) = fold_and_msg_lsb(d_f, d_b, r)
        gb = _read(other, nb.ptr.value, eb.shape, np.uint64)
        gf = _read(other, nf.ptr.value, ef.shape, np.uint64)
        assert (gb == eb).all() and (gf == ef).all()
        assert (u0 == e0).all() and (u2 == e2).all()


@pytest.mark.parametrize("log_n,fails", [(1, False), (2, False), (6, False), (12, False),
                                         (12, True)])
def test_leaves_reused_on_another_stream(ctx, other, log_n, fails):
    """A proof folds in its leaves buffer; what another stream writes there as
    soon as the call returns stays."""
    from bitz_gb300 import DeviceArray, _lib, lib
    from bitz_gb300 import gkr as K
    from oracle import gkr as G

    rng = np.random.default_rng(log_n)
    n = 1 << log_n
    leaves, marks = (rng.integers(0, 2**64, (n, 2), dtype=np.uint64) for _ in range(2))

    class Failing(G.HashChallenges):
        def challenge(self, stage):
            if fails and len(self.messages) > 20:
                raise RuntimeError("no challenge")
            return super().challenge(stage)

    d = DeviceArray.from_host(leaves, ctx)
    for _ in range(16):
        assert lib().bz_memcpy_h2d(ctx.handle, d.ptr, _lib.ptr(leaves), leaves.nbytes) == 0
        if fails:
            with pytest.raises(RuntimeError):
                K.prove(d, 1, [], Failing(b"reuse"), ctx)
        else:
            K.prove(d, 1, [], Failing(b"reuse"), ctx)
        assert lib().bz_memcpy_h2d(other.handle, d.ptr, _lib.ptr(marks), marks.nbytes) == 0
        assert lib().bz_ctx_synchronize(ctx.handle) == 0
        assert (_read(other, d.ptr.value, marks.shape, np.uint64) == marks).all()
