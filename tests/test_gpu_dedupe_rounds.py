"""Duplicate removal where different records share a hash, which takes more
rounds, and at the edges of the hash's and the comparison's segments. The hash
adds, per 8 bytes, the product of two 4-byte halves, each XORed with a constant
of its position: a second half equal to its constant makes the product 0
whatever the first half holds, so records that differ only there collide."""
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


def _half(q):  # the second half of group q that makes its product 0
    return ((q * 0x85EBCA6B + 0x165667B1) & 0xFFFFFFFF).to_bytes(4, "little")


def _colliding(L, q, kinds):
    """`kinds` records of L bytes that differ in the first half of group q."""
    rng = np.random.default_rng(L + q)
    body = bytearray(rng.choice(np.frombuffer(b"ACGT-", np.uint8), L).tobytes())
    body[8 * q + 4:8 * q + 8] = _half(q)
    out = []
    for k in range(kinds):
        body[8 * q:8 * q + 4] = b"%04d" % k
        out.append(bytes(body))
    return out


def _fasta(recs):
    return b"".join(b">" + b"h" * (k % 16) + b"\n" + s + b"\n" for k, s in enumerate(recs))


@pytest.mark.parametrize("L,q", [(8, 0), (11, 0), (512, 62), (4096, 510), (4111, 512), (9000, 1030)])
@pytest.mark.parametrize("kinds", [2, 5])
def test_collisions(ctx, L, q, kinds):
    assert not set(_half(q)) & {10, 13}
    recs = _colliding(L, q, kinds)
    rng = np.random.default_rng(kinds)
    rows = [recs[i] for i in rng.integers(0, kinds, 40)]
    rows += [bytes(r) for r in rng.choice(np.frombuffer(b"ACGT", np.uint8), (30, L))]
    rows += rows[5:45]
    fa = _fasta(rows)
    np.testing.assert_array_equal(ctx.fasta_sequence_indices(fa), o.fasta_sequence_indices(fa))


@pytest.mark.parametrize("late", [False, True])
def test_collisions_in_parts(tmp_path, monkeypatch, late):
    # colliding records in the first part of a streamed file, or across parts
    monkeypatch.setenv("HAMMINGDIST_STREAM_MIN_BYTES", "0")
    L = 1200
    rng = np.random.default_rng(3)
    rows = [bytes(r) for r in rng.choice(np.frombuffer(b"ACGT", np.uint8), (600, L))]
    bad = _colliding(L, 40, 3)
    for k, at in enumerate((5, 300, 580) if late else (5, 9, 40)):
        rows[at] = bad[k]
        rows[at + 10] = bad[k]
    fa = _fasta(rows)
    want, idx = o.from_fasta_dense(fa, remove_duplicates=True, max_distance=65535, dtype=np.uint16)
    got = hd.from_fasta_large(write(tmp_path, "c.fasta", fa), remove_duplicates=True, use_gpu=True,
                              max_distance=65535)
    np.testing.assert_array_equal(np.asarray(got.lt_array), want)


@pytest.mark.parametrize("n", [1, 2, 31, 255, 256, 257, 1025])
def test_numbering(ctx, n):
    # tiles of 256 records, words of 32: all alike, all different, every third
    rng = np.random.default_rng(n)
    for kind in range(3):
        rows = [bytes(r) for r in rng.choice(np.frombuffer(b"ACGT", np.uint8), (n, 40))]
        if kind == 0:
            rows = [rows[0]] * n
        elif kind == 1:
            rows = [rows[k - k % 3] for k in range(n)]
        fa = _fasta(rows)
        np.testing.assert_array_equal(ctx.fasta_sequence_indices(fa), o.fasta_sequence_indices(fa))
