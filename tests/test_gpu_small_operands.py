"""Operands whose dash blocks are written with the plane blocks (up to 16 MB of
them) and those whose listed chunks' blocks follow: the launches of a first
call, and both kinds in one plan, against the bit-plane engine bit for bit."""
import numpy as np
import pytest

from hammingdist_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture
def ctx(monkeypatch):
    from hammingdist_gb300 import abi

    monkeypatch.setenv("HAMMINGDIST_MMA_MIN_ITEMS", "1")
    c = abi.Context(0)
    yield c
    c.close()


def _alignment(ctx, n, L, seed):
    rows, _, _ = synth.alignment(n, L, p=0.1, seed=seed, dash_max=min(200, L // 4))
    rows[n // 2, L // 2: L // 2 + 9] = ord("-")
    return ctx.alignment_from_sequences([r.tobytes() for r in rows])


def _bit_planes(ctx, monkeypatch, aln):
    monkeypatch.setenv("HAMMINGDIST_KERNEL", "lop3")
    want = ctx.pairwise_lt(aln, dtype=np.uint16, max_distance=65535)
    monkeypatch.delenv("HAMMINGDIST_KERNEL")
    return want


# 16 MB: 87,381 rows of one chunk, 560 of 156
@pytest.mark.parametrize("n,L,launches", [(40, 150, 2), (257, 1273, 2), (559, 29903, 3), (561, 29903, 5)])
def test_launches_of_a_first_call(ctx, monkeypatch, n, L, launches):
    aln = _alignment(ctx, n, L, n)
    before = ctx.kernel_launches
    got = ctx.pairwise_lt(aln, dtype=np.uint16, max_distance=65535)
    # rows and chunk list (or rows, list, listed blocks), distances (and the sums of
    # tiles split along K)
    assert ctx.kernel_launches - before == launches
    np.testing.assert_array_equal(got, _bit_planes(ctx, monkeypatch, aln))


def test_both_kinds_in_one_plan(ctx, monkeypatch):
    alns = [_alignment(ctx, n, L, n + L) for n, L in [(60, 500), (620, 29903), (300, 3000), (900, 20000)]]
    b = ctx.batch()
    for a in alns:
        b.add(a, dtype=np.uint16, max_distance=65535)
    for _ in range(2):
        for a, g in zip(alns, b.run()):
            np.testing.assert_array_equal(g, _bit_planes(ctx, monkeypatch, a))
    b.free()


# 32-bit outputs: column halves while twice the items leave every pair of SMs one at
# most (a few thousand rows), whole items above
@pytest.mark.parametrize("n", [2, 257, 512, 2304, 2560, 2816, 3100])
def test_wide_outputs(ctx, monkeypatch, n):
    aln = _alignment(ctx, n, 450, n)
    got = ctx.pairwise_lt(aln, dtype=np.uint32, max_distance=2**32 - 1)
    monkeypatch.setenv("HAMMINGDIST_KERNEL", "lop3")
    np.testing.assert_array_equal(got, ctx.pairwise_lt(aln, dtype=np.uint32, max_distance=2**32 - 1))


# an operand whose first rows' dash blocks were written for their listed chunks only,
# extended by few rows that have the first '-' of other chunks; and the other way round
@pytest.mark.parametrize("first", [640, 40])
def test_extended_operand(ctx, monkeypatch, first):
    import ctypes

    from hammingdist_gb300 import abi

    n, L = 700, 29903
    rows, _, _ = synth.alignment(n, L, p=0.1, seed=first, dash_max=0)
    rows[: first, 100:140] = ord("-")
    rows[first:, 100:120] = ord("N")
    rows[first + 3, 9000:9300] = rows[first + 9, 29900:] = ord("-")
    # the memory that the operand will take holds dash blocks of '-' in every site
    dirty = ctx.alignment_from_sequences([b"-" * L] * n)
    assert not ctx.pairwise_lt(dirty).any()
    dirty.free()
    aln = ctx.alignment_from_sequences([r.tobytes() for r in rows])
    fn = getattr(abi.lib(), "_ZN2hd14ensure_operandEP6hd_ctxPK12hd_alignmentmP11CUstream_stm")
    fn.restype = ctypes.c_bool
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_void_p, ctypes.c_uint64]
    assert fn(ctx.h, aln.h, first, ctx.stream, n)
    got = ctx.pairwise_lt(aln, dtype=np.uint16, max_distance=65535)
    np.testing.assert_array_equal(got, _bit_planes(ctx, monkeypatch, aln))
