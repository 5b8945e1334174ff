"""Site lists at sites where many rows of two tiles differ from the reference: the
warps of a block share such batches of sites. Against the bit-plane engine bit for
bit, at batches of one to many sites and steps of 128, every kind of entry."""
import numpy as np
import pytest

from hammingdist_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from hammingdist_gb300 import abi

    c = abi.Context(0)
    c.trace(True)
    yield c
    c.close()


# a tile of 224 rows has up to 112 x 112 meetings a site here; 4,096 are shared
@pytest.mark.parametrize("n", [130, 225, 700])
@pytest.mark.parametrize("first,sites", [(0, 1), (100, 31), (96, 33), (1020, 8), (1000, 150), (3, 290)])
@pytest.mark.parametrize("kind", ["half", "clade", "N", "runs of N", "some"])
def test_shared_batches(ctx, monkeypatch, n, first, sites, kind):
    L = 2300
    rng = np.random.default_rng(n + sites)
    rows, _, _ = synth.alignment(n, L, p=5e-3, seed=n + first, n_rate=5e-4, dash_max=40)
    s = slice(first, first + sites)
    other = np.where(rows[0, s] == ord("A"), ord("C"), ord("A"))
    if kind == "clade":  # the same rows at every site
        rows[n // 3: 2 * n // 3, s] = other
    elif kind == "runs of N":
        rows[rng.random(n) < 0.5, s] = ord("N")
    else:
        share = 0.25 if kind == "some" else 0.5
        pick = rng.random((n, sites)) < share
        rows[:, s] = np.where(pick, ord("N") if kind == "N" else other, rows[:, s])
    monkeypatch.setenv("HAMMINGDIST_SITE_LISTS", "1")
    aln = ctx.alignment_from_sequences([r.tobytes() for r in rows])
    got = ctx.pairwise_lt(aln, dtype=np.uint16, max_distance=65535)
    assert "site lists" in ctx.trace_last()
    monkeypatch.setenv("HAMMINGDIST_KERNEL", "lop3")
    np.testing.assert_array_equal(got, ctx.pairwise_lt(aln, dtype=np.uint16, max_distance=65535))
    aln.free()
