"""Line and record tables of the device FASTA parse: newlines at the edges of
the scan's 16-byte slices, 8 KB spans and 64 KB blocks, headers after them,
blank lines at every place, unterminated ends, and inputs with just as many
newlines as the tables are first laid out for, and more. The sequence
indices and the reference distances must equal the oracle's."""
import numpy as np
import pytest

from oracle import hd_oracle as o

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from hammingdist_gb300 import abi

    c = abi.Context(0)
    yield c
    c.close()


def _check(ctx, fa, limits=(0, 1, 3)):
    recs = o.read_fasta(fa)[0]
    ref = b"ACGT" * (max([len(s) for s in recs] + [1]) // 4 + 1)
    np.testing.assert_array_equal(ctx.reference_distances(ref, fa),
                                  o.reference_distances(ref, fa))
    for n in limits:
        np.testing.assert_array_equal(ctx.fasta_sequence_indices(fa, n),
                                      o.fasta_sequence_indices(fa, n))


@pytest.mark.parametrize("end", [b"", b"\n", b"\n\n", b"\n>", b"\n>z\n", b"\n>z\n\nAC"])
@pytest.mark.parametrize("edge", [16, 512, 8192, 65536, 131072])
@pytest.mark.parametrize("shift", [-2, -1, 0, 1])
def test_edges(ctx, edge, shift, end):
    # the newline that ends the first sequence is byte edge + shift
    body = b">a\n" + b"ACGTTGCA-N" * (edge // 10 + 1)
    fa = body[:edge + shift] + b"\n>bb\nAC\n>c\nAC\n>d\nACT" + end
    _check(ctx, fa)


@pytest.mark.parametrize("fa", [
    b"", b"\n", b"A", b">a", b">a\n", b"\n\n", b">a\n\n>b\n\n\n", b"AC\nGT\n>b\nA",
    b">a\n\n\nAC\n>b\n\nAC\n\n\n>c\nA\nC\n>d\n\n\n\nA\n\nC\n", b">a\n>b\nAC\n>c\n>d\nAC",
    b"\n\n>a\nAC\n\n>b\nAC\n>", b">a\r\nAC\r\n>b\r\nAC\r\n",
])
def test_blank_and_empty(ctx, fa):
    _check(ctx, fa)


# n two-line records are about 2 n newlines in 6 n bytes; the tables first
# hold 8,192 and one per 2,048 bytes
@pytest.mark.parametrize("newlines", [8190, 8205, 8206, 8207, 8208, 8209, 20001])
@pytest.mark.parametrize("multi", [False, True])
def test_many_lines(ctx, newlines, multi):
    fa = b""
    k = 0
    rows = []
    while len(rows) < newlines:
        rows.append(b">%d" % (k % 10))
        rows.append(b"ACGT"[k % 4:] + b"AAA"[:k % 4])
        if multi and k % 3 == 0:
            rows += [b"", b"G"]
        k += 1
    fa = b"\n".join(rows[:newlines]) + b"\n"
    _check(ctx, fa, (0, 700))
