"""The group passes (ntt_group.cu) and the strided first pass against the
oracle's codeword and against the generic one-layer kernels.

The shapes are the edges of the dispatch: the fewest layers, leftovers of one
and two layers, blocks smaller than a CTA (2 to 8 log lanes, offsets of one to
seven bits), lanes below and above a CTA's threads, the widths of the deepest
tables (k_code 9 .. 18) and first passes strided over 2, 4 and 8 blocks.
Field elements are compared for equality."""
import pytest

pytestmark = pytest.mark.gpu

GENERIC = 0x20
ORACLE = [  # (log_msg_len, log_inv_rate, log_batch_size)
    (3, 1, 1), (5, 1, 2), (7, 1, 2), (8, 2, 3), (9, 1, 1), (10, 1, 0), (10, 2, 4), (11, 1, 3),
    (12, 1, 5), (12, 3, 9), (13, 1, 4), (13, 1, 9), (14, 1, 8), (14, 2, 6), (14, 1, 10),
    (15, 1, 7), (16, 2, 9),
]
GENERIC_SHAPES = [(17, 1, 5), (18, 1, 4), (19, 1, 2), (19, 2, 3), (18, 3, 6), (20, 1, 8),
                  (20, 3, 9), (21, 1, 9), (20, 1, 0), (22, 2, 12), (21, 1, 4), (19, 1, 1)]


def _params(lm, r, lb):
    from bitz_gb300 import PcsParams

    return PcsParams(lm + 7, r, lb, 1)


@pytest.mark.parametrize("lm,r,lb", ORACLE)
def test_default_codeword_equals_oracle(oracle, ctx, lm, r, lb):
    from bitz_gb300 import commit

    msg = oracle.chacha_words(lm * 31 + lb, 1 << lm)
    cw, _, root = oracle.commit(msg, r, lb, 1, n_threads=8)
    c, pd = commit(msg, _params(lm, r, lb), ctx)
    try:
        assert (pd.codeword == cw).all()
        assert c.root == root
    finally:
        pd.free()


@pytest.mark.parametrize("lm,r,lb", GENERIC_SHAPES)
def test_default_equals_generic_layers(lm, r, lb):
    from bitz_gb300 import Context, DeviceArray, commit

    own = Context(0)
    try:
        p = _params(lm, r, lb)
        msg = DeviceArray.chacha(lm + lb, 1 << lm, own)
        c1, d1 = commit(msg, p, own)
        own.set_schedule(p, GENERIC)
        c2, d2 = commit(msg, p, own)
        assert c1.root == c2.root
        assert (d1.codeword == d2.codeword).all()
    finally:
        own.close()
