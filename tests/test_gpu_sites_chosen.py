"""That the site lists compute what they are meant to (the trace names the phase
that builds them), and the choice between them and the tensor cores from a sample
of the sites: both against the bit-plane engine bit for bit."""
import os

import numpy as np
import pytest

from hammingdist_gb300 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture
def ctx():
    from hammingdist_gb300 import abi

    c = abi.Context(0)
    c.trace(True)
    yield c
    c.close()


def _listed(ctx, aln, dtype=np.uint16):
    """(distances, whether the site lists computed them)"""
    out = ctx.pairwise_lt(aln, dtype=dtype, max_distance=np.iinfo(dtype).max)
    return out, "site lists" in ctx.trace_last()


def _bit_planes(ctx, monkeypatch, aln, dtype=np.uint16):
    monkeypatch.setenv("HAMMINGDIST_KERNEL", "lop3")
    out, listed = _listed(ctx, aln, dtype)
    monkeypatch.delenv("HAMMINGDIST_KERNEL")
    assert not listed
    return out


def _pack(ctx, rows, **kw):
    return ctx.alignment_from_sequences([r.tobytes() for r in rows], **kw)


def _mixed(n, L, share, seed):
    """Rows of one root, `share` of the sites any of the six symbols or X."""
    rng = np.random.default_rng(seed)
    root = rng.choice(np.frombuffer(b"ACGTN-", np.uint8), L)
    other = rng.choice(np.frombuffer(b"ACGTN-X", np.uint8), (n, L))
    return np.where(rng.random((n, L)) < share, other, root)


# a quarter of the sites differ (most lists of a full tile hold 50,000 entries);
# 40 and 64 ranges of 1,024 sites
@pytest.mark.parametrize("n,L,share", [(223, 1023, 0.2), (224, 1024, 0.2), (225, 1025, 0.2),
                                       (449, 3001, 0.2), (300, 40000, 0.1), (230, 65536, 0.1)])
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.uint32])
def test_lists_compute(ctx, monkeypatch, n, L, share, dtype):
    monkeypatch.setenv("HAMMINGDIST_SITE_LISTS", "1")
    aln = _pack(ctx, _mixed(n, L, share, n))
    got, listed = _listed(ctx, aln, dtype)
    assert listed
    np.testing.assert_array_equal(got, _bit_planes(ctx, monkeypatch, aln, dtype))


@pytest.mark.parametrize("include_x", [False, True])
def test_lists_compute_sparse_rules(ctx, monkeypatch, include_x):
    from hammingdist_gb300 import abi

    monkeypatch.setenv("HAMMINGDIST_SITE_LISTS", "1")
    rows, _, _ = synth.alignment(300, 2500, p=1e-4, seed=3, n_rate=0.0, dash_max=60)
    rows[::40, ::97] = ord("X")
    aln = _pack(ctx, rows, include_x=include_x, semantics=abi.SEM_CPU)
    got, listed = _listed(ctx, aln)
    assert listed
    np.testing.assert_array_equal(got, _bit_planes(ctx, monkeypatch, aln))


# more than 65,535 entries in a list; more than 64 ranges
@pytest.mark.parametrize("n,L,share", [(300, 2048, 1.0), (3, 65537, 0.01)])
def test_what_lists_do_not_hold(ctx, monkeypatch, n, L, share):
    monkeypatch.setenv("HAMMINGDIST_SITE_LISTS", "1")
    aln = _pack(ctx, _mixed(n, L, share, n))
    got, listed = _listed(ctx, aln, np.uint32)
    assert not listed
    np.testing.assert_array_equal(got, _bit_planes(ctx, monkeypatch, aln, np.uint32))


def _sums_fit(rows):
    """Whether twice the largest sum of m over a row, and the sites of code 0, stay
    within 16 bits, with the commonest code of one bit of the (at most 64) rows, or 0
    where more rows have that than this code and '-'."""
    code = np.zeros(256, np.uint8)
    for c, v in zip(b"ACGT-", (1, 2, 4, 8, 15)):
        code[c] = v
    x = code[rows]
    order = np.array([1, 2, 4, 8])  # of equally common codes the first
    count = np.stack([(x == v).sum(0) for v in order])
    r = order[np.argmax(count, axis=0)]
    r[(x == 0).sum(0) > count.max(0) + (x == 15).sum(0)] = 0
    weight = ((x & r) == 0).sum(1) - (r == 0).sum()
    return 2 * int(weight.max()) + int((r == 0).sum()) <= 65535


@pytest.mark.parametrize("kind", ["unlike", "two unlike four", "alike"])
def test_sums_past_16_bits(ctx, monkeypatch, kind):
    # rows unlike one another; two rows unlike four equal ones, in 3/4 of the sites;
    # rows that differ in half of the sites at most
    monkeypatch.setenv("HAMMINGDIST_SITE_LISTS", "1")
    if kind == "two unlike four":
        rng = np.random.default_rng(1)
        rows = rng.choice(np.frombuffer(b"ACGT", np.uint8), (6, 65536))
        rows[3:] = rows[0]
    else:
        rows = _mixed(6, 65536, 1.0 if kind == "unlike" else 0.3, 6)
    aln = _pack(ctx, rows)
    got, listed = _listed(ctx, aln, np.uint32)
    assert listed == _sums_fit(rows) == (kind == "alike")
    np.testing.assert_array_equal(got, _bit_planes(ctx, monkeypatch, aln, np.uint32))


def test_row_ranges_inside_tiles(ctx, monkeypatch, tmp_path):
    # the text of 9,600 rows is written in two ranges of rows of 128; the second
    # starts inside a tile of 224, at a lower-triangle index of its own
    n, L = 9600, 40
    assert n * (n - 1) // 2 * 6 > 256 << 20 and 9344 % 128 == 0 and 9344 % 224
    assert 9344 * 9343 // 2 * 6 <= 256 << 20 < (9344 + 128) * (9344 + 127) // 2 * 6
    aln = _pack(ctx, _mixed(n, L, 0.1, 9))
    text = []
    for env, value in (("HAMMINGDIST_SITE_LISTS", "1"), ("HAMMINGDIST_KERNEL", "lop3")):
        monkeypatch.setenv(env, value)
        if value == "1":
            assert _listed(ctx, aln)[1]  # the lists stay with the alignment
        ctx.pairwise_lt_to_file(aln, 255, str(tmp_path / value))
        monkeypatch.delenv(env)
        text.append((tmp_path / value).read_bytes())
    assert text[0] == text[1]


def _device_rows(ctx, n, L, p):
    text = torch.empty(ctx.synthetic_fasta(n, L, p=p, seed=n), dtype=torch.uint8, device="cuda")
    ctx.synthetic_fasta(n, L, p=p, seed=n, out=text.data_ptr())
    ctx.synchronize()
    return text


# samples of all words, of an eighth and of a sixteenth; sizes just past 0.2 ms of
# the tensor cores, below which nothing is sampled
@pytest.mark.parametrize("n,L", [(10600, 3000), (10100, 8191), (7200, 8193), (5400, 16385),
                                 (4600, 29903)])
@pytest.mark.parametrize("p,alike", [(1e-3, True), (0.1, False)])
@pytest.mark.parametrize("compared", [False, True])
def test_choice_by_a_sample(ctx, monkeypatch, n, L, p, alike, compared):
    text = _device_rows(ctx, n, L, p)
    if compared:
        ctx.expect_pairwise()
    aln = ctx.alignment_from_fasta(text.data_ptr(), text.numel(), on_device=True)
    got, listed = _listed(ctx, aln)
    assert listed == alike
    np.testing.assert_array_equal(got, _bit_planes(ctx, monkeypatch, aln))


@pytest.mark.parametrize("kind", ["alike", "diverse", "diverse from half on"])
def test_choice_of_a_streamed_file(ctx, monkeypatch, tmp_path, kind):
    n, L = 4600, 29903
    text = _device_rows(ctx, n, L, 0.1 if kind == "diverse" else 1e-3).cpu().numpy()
    if kind == "diverse from half on":  # after the sample
        rec = text[: text.size // n * n].reshape(n, -1)
        rng = np.random.default_rng(1)
        rec[n // 2:, -L - 1:-1] = rng.choice(np.frombuffer(b"ACGT", np.uint8), (n - n // 2, L))
    path = str(tmp_path / "s.fasta")
    text.tofile(path)
    got, aln = ctx.pairwise_lt_fasta_file(path, dtype=np.uint16, max_distance=65535)
    trace = ctx.trace_last()
    assert ("site lists built" in trace) == (kind != "diverse")
    np.testing.assert_array_equal(got, _bit_planes(ctx, monkeypatch, aln))
    listed = _listed(ctx, aln)[1]
    assert listed == (kind == "alike")
