"""One alignment, several threads with a context each: what the alignment builds on
first use (the tensor-core operand and its chunk list, the site lists) is built
once and read only when it is there, also by a server's windows. Results equal
those of one context alone."""
import threading

import numpy as np
import pytest

from hammingdist_gb300 import synth

pytestmark = pytest.mark.gpu


def _rows(n, L, seed):
    rows, _, _ = synth.alignment(n, L, p=1e-2, seed=seed, dash_max=min(200, L // 3))
    return rows


def _together(work):
    """Runs the calls at once and returns their results."""
    out, start = [None] * len(work), threading.Barrier(len(work))

    def run(k):
        start.wait()
        try:
            out[k] = work[k]()
        except Exception as e:  # shown by the comparison
            out[k] = e

    th = [threading.Thread(target=run, args=(k,)) for k in range(len(work))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    return out


@pytest.mark.parametrize("engine", ["HAMMINGDIST_SITE_LISTS", "HAMMINGDIST_MMA_MIN_ITEMS"])
def test_first_use_by_several_contexts(monkeypatch, engine):
    from hammingdist_gb300 import abi

    monkeypatch.setenv(engine, "1")
    if engine != "HAMMINGDIST_SITE_LISTS":
        monkeypatch.setenv("HAMMINGDIST_SITE_LISTS", "0")
    ctxs = [abi.Context(0) for _ in range(4)]
    try:
        for k, (n, L) in enumerate([(700, 3000), (300, 20000), (1200, 1000), (600, 29903)]):
            seqs = [r.tobytes() for r in _rows(n, L, k)]
            alone = ctxs[0].alignment_from_sequences(seqs)
            want = ctxs[0].pairwise_lt(alone, dtype=np.uint16, max_distance=65535)
            shared = ctxs[0].alignment_from_sequences(seqs)
            batches = [c.batch() for c in ctxs[2:]]
            for b in batches:  # (the others' plans take one matrix)
                b.add(shared, dtype=np.uint16, max_distance=65535)
                b.add(alone, dtype=np.uint16, max_distance=65535)
            got = _together([lambda c=c: c.pairwise_lt(shared, dtype=np.uint16, max_distance=65535)
                             for c in ctxs[:2]] + [lambda b=b: b.run()[0] for b in batches])
            for g in got:
                np.testing.assert_array_equal(g, want)
            for b in batches:
                b.free()
            shared.free()
            alone.free()
    finally:
        for c in reversed(ctxs):
            c.close()


def test_windows_while_a_call_builds_the_operand(monkeypatch):
    from hammingdist_gb300 import abi

    monkeypatch.setenv("HAMMINGDIST_MMA_MIN_ITEMS", "1")
    monkeypatch.setenv("HAMMINGDIST_SITE_LISTS", "0")
    ctx, other = abi.Context(0), abi.Context(0)
    try:
        n, L = 1500, 20000
        seqs = [r.tobytes() for r in _rows(n, L, 7)]
        first = other.alignment_from_sequences(seqs)
        want = other.pairwise_lt(first, dtype=np.uint16, max_distance=65535)
        for _ in range(3):
            aln = ctx.alignment_from_sequences(seqs)
            srv = ctx.server()
            ident = srv.add(aln)
            windows = [(0, 300), (0, n), (5, 200), (0, 1000)] * 3

            def serve():
                t = [srv.pairwise(ident, r0, m, dtype=np.uint16, max_distance=65535) for r0, m in windows]
                for q in t:
                    srv.wait(q)
                return [srv.result(q)[0] for q in t]

            served, plain = _together(
                [serve, lambda: other.pairwise_lt(aln, dtype=np.uint16, max_distance=65535)])
            np.testing.assert_array_equal(plain, want)
            i, j = np.tril_indices(n, -1)
            for (r0, m), g in zip(windows, served):
                rows = slice(r0, r0 + m)
                full = np.zeros((n, n), np.uint16)
                full[i, j] = want
                a, b = np.tril_indices(m, -1)
                np.testing.assert_array_equal(g, full[rows, rows][a, b])
            srv.free()
            aln.free()
        first.free()
    finally:
        other.close()
        ctx.close()
