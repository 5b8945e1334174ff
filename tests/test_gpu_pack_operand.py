"""Rows packed together with their tensor-core operand (expect_pairwise), at
the edges of words, chunks and vectors and with every byte value, against the
oracle; and operands that grow part by part, whose chunks get their first '-'
in any part."""
import numpy as np
import pytest

from gpu_util import write
from oracle import hd_oracle as o

pytestmark = pytest.mark.gpu
hd = pytest.importorskip("hammingdist_gb300")


@pytest.fixture(scope="module")
def ctx():
    from hammingdist_gb300 import abi

    c = abi.Context(0)
    yield c
    c.close()


def _fasta(rows):
    # headers of 2 to 17 bytes: every alignment of a row's first byte
    return b"".join(b">" + b"h" * (k % 16) + b"\n" + r.tobytes() + b"\n"
                    for k, r in enumerate(rows))


@pytest.mark.parametrize("L", [1, 7, 31, 32, 33, 191, 192, 193, 255, 257, 383, 385, 1537])
@pytest.mark.parametrize("symbols", ["ACGT", "ACGT-", "bytes"])
@pytest.mark.parametrize("n", [2, 17, 129])
def test_pack_with_operand(ctx, monkeypatch, L, symbols, n):
    monkeypatch.setenv("HAMMINGDIST_MMA_MIN_ITEMS", "0")
    rng = np.random.default_rng(L * 1000 + n)
    if symbols == "bytes":  # every value but the line ends, and '>' first in a line
        pool = np.array([b for b in range(256) if b not in (10, 13, ord(">"))], np.uint8)
        pool = np.concatenate([pool, np.frombuffer(b"ACGT-" * 60, np.uint8)])
    else:
        pool = np.frombuffer(symbols.encode(), np.uint8)
    rows = rng.choice(pool, (n, L))
    rows[n // 2] = rows[0]
    fa = _fasta(rows)
    for dup in (False, True):
        want, idx = o.from_fasta_dense(fa, remove_duplicates=dup, max_distance=65535,
                                       dtype=np.uint16)
        ctx.expect_pairwise()
        a = ctx.alignment_from_fasta(fa, remove_duplicates=dup)
        got = ctx.pairwise_lt(a, dtype=np.uint16, max_distance=65535)
        np.testing.assert_array_equal(got, want)
        monkeypatch.setenv("HAMMINGDIST_KERNEL", "lop3")  # the packed rows themselves
        np.testing.assert_array_equal(ctx.pairwise_lt(a, dtype=np.uint16, max_distance=65535), want)
        monkeypatch.delenv("HAMMINGDIST_KERNEL")
        a.free()


@pytest.mark.parametrize("where", [[], [0], [600], [899], [0, 330, 600, 899], list(range(0, 900, 7))])
@pytest.mark.parametrize("dup", [False, True])
def test_growing_operand(tmp_path, monkeypatch, where, dup):
    # three parts of about 300 rows; the rows `where` have '-' in other chunks
    # each, so chunks are first marked by any of the parts
    monkeypatch.setenv("HAMMINGDIST_MMA_MIN_ITEMS", "0")
    monkeypatch.setenv("HAMMINGDIST_STREAM_MIN_BYTES", "0")
    rng = np.random.default_rng(len(where))
    rows = rng.choice(np.frombuffer(b"ACGTN", np.uint8), (900, 1200))
    for k, r in enumerate(where):
        rows[r, (k * 200) % 1200:(k * 200) % 1200 + 30] = ord("-")
    rows[450] = rows[3]
    fa = _fasta(rows)
    want, idx = o.from_fasta_dense(fa, remove_duplicates=dup, max_distance=65535, dtype=np.uint16)
    got = hd.from_fasta_large(write(tmp_path, "g.fasta", fa), remove_duplicates=dup, use_gpu=True,
                              max_distance=65535)
    np.testing.assert_array_equal(np.asarray(got.lt_array), want)
