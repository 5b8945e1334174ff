"""Distances from site lists against the bit-plane engine bit for bit (whole
numbers: no tolerance): tiles of 224 rows, ranges of 1,024 sites, 32-entry
chunks and long lists at their edges, every kind of site, all rules, types and
caps, and rows too different or too many for the lists."""
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


def _both(ctx, monkeypatch, rows, dtype, md, **kw):
    monkeypatch.setenv("HAMMINGDIST_SITE_LISTS", "1")
    aln = ctx.alignment_from_sequences([r.tobytes() for r in rows], **kw)
    got = ctx.pairwise_lt(aln, dtype=dtype, max_distance=md)
    monkeypatch.setenv("HAMMINGDIST_KERNEL", "lop3")
    want = ctx.pairwise_lt(aln, dtype=dtype, max_distance=md)
    monkeypatch.delenv("HAMMINGDIST_KERNEL")
    aln.free()
    np.testing.assert_array_equal(got, want)


def _rows(n, L, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "random":
        return rng.choice(np.frombuffer(b"ACGTN-X", np.uint8), (n, L))
    rows, _, _ = synth.alignment(n, L, p=1e-2, seed=seed, n_rate=1e-3, dash_max=min(200, L // 4))
    if kind == "columns":  # sites of one symbol, of two halves, and of N but for a few rows
        at = rng.permutation(L)[:max(1, L // 8)]
        for q, c in enumerate(at):
            rows[:, c] = ord("N-XAC"[q % 5])
            if q % 3 == 1:
                rows[: n // 2, c] = ord("G")
            elif q % 3 == 2:
                rows[rng.integers(0, n), c] = ord("ACGT-N"[q % 6])
    return rows


@pytest.mark.parametrize("n,L", [(2, 1), (3, 31), (223, 1023), (224, 1024), (225, 1025),
                                 (449, 3001), (700, 2048)])
@pytest.mark.parametrize("kind", ["alike", "columns", "random"])
@pytest.mark.parametrize("dtype,md", [(np.uint8, 255), (np.uint8, 9), (np.uint16, 65535),
                                      (np.uint32, 2**32 - 1)])
def test_dense_rule(ctx, monkeypatch, n, L, kind, dtype, md):
    _both(ctx, monkeypatch, _rows(n, L, kind, n + L), dtype, md)


@pytest.mark.parametrize("include_x", [False, True])
@pytest.mark.parametrize("n,L", [(225, 1025), (300, 4000)])
def test_sparse_rules(ctx, monkeypatch, include_x, n, L):
    from hammingdist_gb300 import abi

    rows, _, _ = synth.alignment(n, L, p=1e-4, seed=n, n_rate=0.0, dash_max=60)
    rows[::40, ::97] = ord("X")
    rows[7, 100:160] = ord("N")
    _both(ctx, monkeypatch, rows, np.uint16, 65535, include_x=include_x, semantics=abi.SEM_CPU)


def test_weights_past_16_bits(ctx, monkeypatch):
    # rows that differ from the reference in more than half of 65,536 sites
    rng = np.random.default_rng(1)
    rows = rng.choice(np.frombuffer(b"ACGT", np.uint8), (6, 65536))
    rows[3:] = rows[0]
    _both(ctx, monkeypatch, rows, np.uint32, 2**32 - 1)
    _both(ctx, monkeypatch, rng.choice(np.frombuffer(b"ACGT", np.uint8), (3, 65537)), np.uint32,
          2**32 - 1)


def test_file_in_row_ranges(ctx, monkeypatch, tmp_path):
    # the writer's row ranges start inside tiles
    rows = _rows(1500, 1100, "alike", 5)
    monkeypatch.setenv("HAMMINGDIST_SITE_LISTS", "1")
    aln = ctx.alignment_from_sequences([r.tobytes() for r in rows])
    ctx.pairwise_lt_to_file(aln, 255, str(tmp_path / "a.txt"))
    monkeypatch.setenv("HAMMINGDIST_KERNEL", "lop3")
    ctx.pairwise_lt_to_file(aln, 255, str(tmp_path / "b.txt"))
    monkeypatch.delenv("HAMMINGDIST_KERNEL")
    aln.free()
    assert (tmp_path / "a.txt").read_bytes() == (tmp_path / "b.txt").read_bytes()


@pytest.mark.parametrize("n,L,kind", [(1600, 8300, "alike"), (1100, 45000, "random4")])
@pytest.mark.parametrize("dup", [False, True])
def test_streamed_file(tmp_path, monkeypatch, n, L, kind, dup):
    # the lists of a file's parts, and a file whose rows turn out too different
    hd = pytest.importorskip("hammingdist_gb300")
    from gpu_util import write

    rng = np.random.default_rng(n)
    rows = (rng.choice(np.frombuffer(b"ACGT", np.uint8), (n, L)) if kind == "random4"
            else _rows(n, L, kind, 3))
    rows[n // 2:n // 2 + 40] = rows[:40]
    path = write(tmp_path, "s.fasta", synth.to_fasta(rows))
    monkeypatch.setenv("HAMMINGDIST_STREAM_MIN_BYTES", "0")
    got = []
    for env in ("HAMMINGDIST_SITE_LISTS", "HAMMINGDIST_KERNEL"):
        monkeypatch.setenv(env, {"HAMMINGDIST_KERNEL": "lop3"}.get(env, "1"))
        ds = hd.from_fasta_large(path, remove_duplicates=dup, use_gpu=True)
        got.append(np.array(ds.lt_array))
        monkeypatch.delenv(env)
        os.utime(path, ns=(1, len(got)))  # read again, not the file already on the device
    np.testing.assert_array_equal(got[0], got[1])
