"""Edges of the opening's table kernels against the oracle, for equality: eq
tables around the switch to rows of byte-table products, the ring switch's
bit sums at lengths that leave part of a tile, a warp or a group of four
words, and the out-of-domain sample around the switch to column sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rand(seed, n):
    return np.random.default_rng(seed).integers(0, 2**64, (n, 2), dtype=np.uint64)


@pytest.mark.parametrize("k", [8, 11, 16, 17, 18, 19, 21])
def test_build_eq_rows(oracle, ctx, k):
    from bitz_gb300.ligerito import build_eq_lsb

    pt = _rand(500 + k, k)
    assert (build_eq_lsb(pt, ctx).to_host() == oracle.build_eq_lsb(pt)).all()


@pytest.mark.parametrize("n", [1, 3, 4, 31, 33, 127, 128, 129, 1000, 6 * 152 * 128 + 37])
def test_sv_fold_ragged(oracle, ctx, n):
    from bitz_gb300 import DeviceArray
    from bitz_gb300.ligerito import sv_fold

    P, eq = _rand(n, n), _rand(n + 1, n)
    got = sv_fold(DeviceArray.from_host(P, ctx), DeviceArray.from_host(eq, ctx))
    assert (got == oracle.sv_fold(P, eq)).all()


@pytest.mark.parametrize("m", [11, 14, 15, 18, 21])
def test_round0_rows(oracle, ctx, m):
    from bitz_gb300 import BinaryPcs, Blake3Transcript, DeviceArray, LigeritoConfig
    from oracle.binary_pcs import prove_round0
    from oracle.transcript import Blake3Transcript as OT

    packed = oracle.chacha_words(m + 40, 1 << m)
    exp = prove_round0(OT(), packed, 0)
    d = DeviceArray.from_host(packed, ctx)
    try:
        pcs = BinaryPcs(m, LigeritoConfig(1, [0], [1, 1], [1, 1], [0, 0]), 0, ctx)
        got = pcs.prove_round0(Blake3Transcript(), d)
        assert got.y.tolist() == exp.y.tolist()
    finally:
        d.free()
