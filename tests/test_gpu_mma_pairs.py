"""The tensor-core engine's items (256 rows x 496 columns on a pair of SMs,
192-site chunks) at their edges, and tiles split along K, against the
bit-plane engine bit for bit (whole numbers: no tolerance)."""
import os

import numpy as np
import pytest

from hammingdist_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from hammingdist_gb300 import abi

    c = abi.Context(0)
    yield c
    c.close()


# rows around one and two items and their column halves; lengths around one
# chunk, a few chunks, and many chunks of few tiles (every tile in K pieces)
@pytest.mark.parametrize("n,L", [(255, 287), (256, 288), (257, 289), (272, 576), (496, 577),
                                 (497, 1152), (513, 2881), (753, 3000), (130, 20000),
                                 (500, 29903), (1009, 14401)])
@pytest.mark.parametrize("dtype,md", [(np.uint8, 255), (np.uint16, 65535), (np.uint16, 700),
                                      (np.uint32, 2**32 - 1)])
def test_pair_items(ctx, monkeypatch, n, L, dtype, md):
    monkeypatch.setenv("HAMMINGDIST_MMA_MIN_ITEMS", "0")
    rows, _, _ = synth.alignment(n, L, p=0.2, seed=n + L, dash_max=min(200, L // 3))
    aln = ctx.alignment_from_sequences([r.tobytes() for r in rows])
    got = ctx.pairwise_lt(aln, dtype=dtype, max_distance=md)
    os.environ["HAMMINGDIST_KERNEL"] = "lop3"
    try:
        want = ctx.pairwise_lt(aln, dtype=dtype, max_distance=md)
    finally:
        del os.environ["HAMMINGDIST_KERNEL"]
    np.testing.assert_array_equal(got, want)
    aln.free()


def test_small_batch_splits_along_k(ctx):
    # a batch of few, long matrices: the queue's items are cut along K, and
    # the 6-plane rule's two dash blocks fall into several pieces
    from hammingdist_gb300 import abi

    sets = []
    for k, (n, L) in enumerate([(300, 29903), (140, 14000), (260, 20011)]):
        rows, _, _ = synth.alignment(n, L, p=1e-4, seed=k, n_rate=0.0)
        rows[::40, ::97] = ord("X")
        sets.append(ctx.alignment_from_sequences([r.tobytes() for r in rows], include_x=True,
                                                 semantics=abi.SEM_CPU))
    b = ctx.batch()
    for a in sets:
        b.add(a, dtype=np.uint16, max_distance=65535)
    first = b.run()
    again = b.run()  # the replayed graph
    os.environ["HAMMINGDIST_KERNEL"] = "lop3"
    try:
        want = [ctx.pairwise_lt(a, dtype=np.uint16, max_distance=65535) for a in sets]
    finally:
        del os.environ["HAMMINGDIST_KERNEL"]
    for f, g, w in zip(first, again, want):
        np.testing.assert_array_equal(f, w)
        np.testing.assert_array_equal(g, w)
    b.free()
    for a in sets:
        a.free()
