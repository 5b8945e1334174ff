"""Operands of several matrices of one plan: their chunk lists and dash blocks are
made together, one launch for each matrix's rows and a fixed number for all, and
every result equals the bit-plane engine's."""
import numpy as np
import pytest

from hammingdist_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture
def ctx():
    from hammingdist_gb300 import abi

    c = abi.Context(0)
    yield c
    c.close()


def _rows(n, L, seed):
    """Rows with '-' in some chunks of 192 sites only: none, the ends, one row's middle."""
    rows, _, _ = synth.alignment(n, L, p=2e-2, seed=seed, n_rate=1e-3,
                                 dash_max=(0, min(60, L // 4), 0)[seed % 3])
    if seed % 3 == 2 and n > 1:
        rows[n - 1, L // 2: L // 2 + 5] = ord("-")
    return rows


SIZES = [(2, 5), (9, 192), (30, 193), (64, 577), (129, 3001), (257, 1000), (500, 2100), (17, 8000)]


@pytest.mark.parametrize("rule", ["dense", "sparse", "sparse_x"])
def test_batch_equals_bit_planes(ctx, monkeypatch, rule):
    from hammingdist_gb300 import abi

    kw = {} if rule == "dense" else {"include_x": rule == "sparse_x", "semantics": abi.SEM_CPU}
    monkeypatch.setenv("HAMMINGDIST_MMA_MIN_ITEMS", "1")
    alns, want = [], []
    for k, (n, L) in enumerate(SIZES + SIZES[:3]):
        rows = _rows(n, L, k)
        if rule == "sparse":
            rows[:] = np.where(rows == ord("-"), rows, rows[0])  # alike: the sparse rule is chosen
        alns.append(ctx.alignment_from_sequences([r.tobytes() for r in rows], **kw))
    alns.append(alns[4])  # one alignment twice
    monkeypatch.setenv("HAMMINGDIST_KERNEL", "lop3")
    want = [ctx.pairwise_lt(a, dtype=np.uint16, max_distance=65535) for a in alns]
    monkeypatch.delenv("HAMMINGDIST_KERNEL")
    b = ctx.batch()
    for a in alns:
        b.add(a, dtype=np.uint16, max_distance=65535)
    for _ in range(2):  # planned, then replayed
        for g, w in zip(b.run(), want):
            np.testing.assert_array_equal(g, w)
    # the operands stay: the same alignments alone
    for a, w in zip(alns, want):
        np.testing.assert_array_equal(ctx.pairwise_lt(a, dtype=np.uint16, max_distance=65535), w)
    b.free()


def test_one_launch_for_each_operand(ctx, monkeypatch):
    monkeypatch.setenv("HAMMINGDIST_MMA_MIN_ITEMS", "1")
    jobs = 40
    alns = [ctx.alignment_from_sequences([r.tobytes() for r in _rows(20 + k, 300, k)])
            for k in range(jobs)]
    b = ctx.batch()
    for a in alns:
        b.add(a)
    before = ctx.kernel_launches
    b.run()
    assert jobs < ctx.kernel_launches - before <= jobs + 8
    b.free()
