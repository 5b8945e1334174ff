"""The reference of the site lists at sites where the rows it is taken from have
'-' or 'N' only: the '-' of all other rows stay '-' entries there, so that the
lists hold them, and the distances are the bit-plane engine's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65, 159, 160, 161, 255, 256, 257, 700])
@pytest.mark.parametrize("seen", [b"N", b"-", b"NN-"])
def test_ends_that_few_rows_reach(monkeypatch, n, seen):
    from hammingdist_gb300 import abi

    L, ends = 1024, 200
    rng = np.random.default_rng(n)
    acgt = np.frombuffer(b"ACGT", np.uint8)
    root = rng.choice(acgt, L)
    rows = np.where(rng.random((n, L)) < 0.16, rng.choice(acgt, (n, L)), root)
    rows[:, :ends] = ord("-")
    reach = rng.choice(n, max(2, n // 20), replace=False)  # rows that have the end
    rows[reach, :ends] = root[:ends]
    looked_at = [n * q // 64 for q in range(64)]
    rows[looked_at, :ends] = ord("-")
    for k, c in enumerate(seen):
        rows[looked_at[k], :ends] = c
    monkeypatch.setenv("HAMMINGDIST_SITE_LISTS", "1")
    ctx = abi.Context(0)
    try:
        ctx.trace(True)
        aln = ctx.alignment_from_sequences([r.tobytes() for r in rows])
        got = ctx.pairwise_lt(aln, dtype=np.uint16, max_distance=65535)
        # as s entries the '-' of a tile of 224 rows would be 44,800 with 29,000 others
        assert "site lists" in ctx.trace_last()
        monkeypatch.setenv("HAMMINGDIST_KERNEL", "lop3")
        np.testing.assert_array_equal(got, ctx.pairwise_lt(aln, dtype=np.uint16, max_distance=65535))
        aln.free()
    finally:
        ctx.close()


@pytest.mark.parametrize("n", [5, 64, 300])
def test_sites_of_n(monkeypatch, n):
    # sites where most rows have 'N', all of them, or half of them and half '-'
    from hammingdist_gb300 import abi

    rng = np.random.default_rng(n)
    rows = np.tile(rng.choice(np.frombuffer(b"ACGT", np.uint8), 2100), (n, 1))
    for k, share in enumerate((1.0, 0.8, 0.5, 0.3)):
        for j, other in enumerate((None, ord("-"), ord("A"))):
            s = slice(1000 + 40 * (3 * k + j), 1000 + 40 * (3 * k + j) + 33)
            pick = rng.random(n) < share
            rows[pick, s] = ord("N")
            if other:
                rows[~pick, s] = other
    monkeypatch.setenv("HAMMINGDIST_SITE_LISTS", "1")
    ctx = abi.Context(0)
    try:
        ctx.trace(True)
        aln = ctx.alignment_from_sequences([r.tobytes() for r in rows])
        got = ctx.pairwise_lt(aln, dtype=np.uint16, max_distance=65535)
        assert "site lists" in ctx.trace_last()
        monkeypatch.setenv("HAMMINGDIST_KERNEL", "lop3")
        np.testing.assert_array_equal(got, ctx.pairwise_lt(aln, dtype=np.uint16, max_distance=65535))
        aln.free()
    finally:
        ctx.close()
