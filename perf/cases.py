"""Performance cases: the work that users of this framework have it do.

Each case is a dict of plain values; `prepare` builds what a program has in
hand before the call (files, resident buffers, packed alignments), `run` makes
one pass through the public entry points and returns its results whole.

Sequences follow the model of hammingdist_gb300/synth.py: a root uniform over
ACGT, substitutions with probability p per site, N runs of 1-50 sites (about
1e-4 per site), leading and trailing '-' runs of up to 200 sites (up to L/8
for short rows), and exact duplicates of earlier records. Record headers are
sized so that records start at every byte alignment. Files live in memory
(memfd), as a file in the page cache does, without writeback disturbing the
passes.
"""
import math
import os

import numpy as np
import torch

import hammingdist_gb300 as hd
from hammingdist_gb300 import abi

DEV = "cuda"
_ACGT = torch.tensor(list(b"ACGT"), dtype=torch.uint8)


def listed():
    return [
        # one pair of genomes: the smallest call there is, all latency
        {"name": "distance pair", "kind": "distance", "L": 29903, "p": 0.2},
        # a list of short sequences from a notebook, the default (CPU) semantics
        {"name": "stringlist", "kind": "strings", "n": 120, "L": 1273, "p": 2e-2},
        # a small outbreak file, GPU semantics (the reference's small configuration)
        {"name": "file 1k", "kind": "file", "n": 1000, "L": 29903, "p": 1e-3, "dup": 0.0,
         "use_gpu": True, "include_x": False, "wide": False, "refs": False},
        # from_fasta's default call (CPU semantics) on a low-diversity set
        {"name": "file cpu semantics", "kind": "file", "n": 3001, "L": 29903, "p": 1e-3, "dup": 0.2,
         "use_gpu": False, "include_x": False, "wide": False, "refs": False},
        # the headline call: a large file with duplicates, then the root's
        # distances from the same file
        {"name": "file 20k", "kind": "file", "n": 20000, "L": 29903, "p": 1e-3, "dup": 0.3,
         "use_gpu": True, "include_x": False, "wide": False, "refs": True},
        # the same work on FASTA text already in HBM, result left there
        {"name": "device 20k", "kind": "device", "n": 20000, "L": 29903, "p": 1e-3, "dup": 0.3,
         "wide": False},
        # distances of a large packed alignment that stays on the device
        {"name": "resident 14k", "kind": "resident", "n": 14001, "L": 29903, "p": 1e-3, "bytes": 1},
        # short rows (one gene), wide distances
        {"name": "resident short", "kind": "resident", "n": 1500, "L": 1273, "p": 2e-2, "bytes": 2},
        # uneven alignments computed together from device-resident rows
        {"name": "batch", "kind": "batch", "jobs": 48, "n_lo": 50, "n_hi": 5000, "p": 1e-3},
        # a new sequence against a resident set (serving's commonest request)
        {"name": "query 50k", "kind": "query", "n": 50000, "L": 29903, "p": 1e-3},
        # the lower-triangular text of a large matrix
        {"name": "text 14k", "kind": "text", "n": 14000, "bytes": 1, "mean": 60},
        # distances computed earlier, read back from such a file
        {"name": "read 9k", "kind": "read", "n": 9001, "bytes": 1, "mean": 60, "csv": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cap_rows(n, L, most):
    """n, lowered so that n^2 L stays within `most`."""
    return max(2, min(n, int(math.sqrt(most / L))))


def draw(rng):
    kind = rng.choice(["distance", "strings", "file", "file", "device", "resident", "resident",
                       "batch", "query", "text", "read"])
    p = math.exp(rng.uniform(math.log(1e-4), math.log(3e-2)))
    if kind == "distance":
        return {"kind": kind, "L": _log(rng, 1000, 60000), "p": rng.uniform(0.05, 0.75)}
    if kind == "strings":
        return {"kind": kind, "n": _log(rng, 8, 400), "L": _log(rng, 100, 3000), "p": max(p, 1e-2)}
    if kind == "file":
        L = _log(rng, 300, 40000)
        n = _cap_rows(_log(rng, 50, 20000), L, 14000.0 ** 2 * 29903)
        n = min(n, int(590e6 / (L + 13)))
        use_gpu = rng.random() < 0.6
        include_x = not use_gpu and rng.random() < 0.3
        if not use_gpu:
            n = min(n, 6000)
        return {"kind": kind, "n": n, "L": L, "p": p, "dup": rng.choice([0.0, 0.1, 0.3]),
                "use_gpu": use_gpu, "include_x": include_x, "wide": rng.random() < 0.3,
                "refs": rng.random() < 0.5}
    if kind == "device":
        L = _log(rng, 300, 40000)
        n = _cap_rows(_log(rng, 100, 20000), L, 14000.0 ** 2 * 29903)
        return {"kind": kind, "n": n, "L": L, "p": p, "dup": rng.choice([0.0, 0.3]),
                "wide": rng.random() < 0.3}
    if kind == "resident":
        L = _log(rng, 100, 60000)
        n = _cap_rows(_log(rng, 100, 16000), L, 14000.0 ** 2 * 29903)
        return {"kind": kind, "n": n, "L": L, "p": p, "bytes": rng.choice([1, 1, 2, 4])}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(4, 60), "n_lo": _log(rng, 20, 100),
                "n_hi": _log(rng, 300, 5000), "p": p}
    if kind == "query":
        return {"kind": kind, "n": _log(rng, 500, 50000), "L": _log(rng, 300, 30000), "p": p}
    if kind == "text":
        return {"kind": kind, "n": _log(rng, 300, 14000), "bytes": rng.choice([1, 2, 4]),
                "mean": rng.choice([5, 60, 200])}
    csv = rng.random() < 0.4
    return {"kind": kind, "n": _log(rng, 300, 6000 if csv else 9000),
            "bytes": 1 if csv else rng.choice([1, 2]), "mean": rng.choice([5, 60, 200]), "csv": csv}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _root(L, g):
    return _ACGT.to(DEV)[torch.randint(0, 4, (L,), device=DEV, generator=g)]


def _rows(n, L, p, g, root):
    """n mutated copies of root: uint8 [n, L]."""
    x = root.expand(n, L).contiguous()
    flat = x.view(-1)
    k = int(n * L * p)
    if k:
        at = torch.unique(torch.randint(0, n * L, (k,), device=DEV, generator=g))
        flat[at] = _ACGT.to(DEV)[torch.randint(0, 4, (at.numel(),), device=DEV, generator=g)]
    runs = int(n * L * 1e-4)
    if runs:
        start = torch.randint(0, n * L, (runs,), device=DEV, generator=g)
        length = torch.randint(1, 51, (runs,), device=DEV, generator=g)
        end = torch.minimum(start + length, (start // L + 1) * L)
        for o in range(50):
            at = start + o
            flat[at[at < end]] = ord("N")
    most = min(200, L // 8)
    if most:
        col = torch.arange(L, device=DEV, dtype=torch.int32)
        lead = torch.randint(0, most + 1, (n, 1), device=DEV, generator=g, dtype=torch.int32)
        trail = torch.randint(0, most + 1, (n, 1), device=DEV, generator=g, dtype=torch.int32)
        for r in range(0, n, 2048):
            s = slice(r, r + 2048)
            x[s].masked_fill_((col < lead[s]) | (col >= L - trail[s]), ord("-"))
    return x


def _records(case, seed):
    """(rows uint8 [n, L] on the device, root): the records of a file, duplicates included."""
    g = _gen(seed)
    n, L = case["n"], case["L"]
    root = _root(L, g)
    dups = int(n * case.get("dup", 0.0))
    x = _rows(n - dups, L, case["p"], g, root)
    if dups:
        rng = np.random.default_rng(int(seed))
        is_dup = np.zeros(n, dtype=bool)
        is_dup[rng.choice(np.arange(1, n), size=dups, replace=False)] = True
        first = np.cumsum(~is_dup) - 1
        src = np.where(is_dup, (rng.random(n) * (first + 1)).astype(np.int64), first)
        x = x[torch.from_numpy(src).to(DEV)]
    return x, root


def _fasta(x):
    """The FASTA text of rows x, as a device tensor."""
    n, L = x.shape
    digits = len(str(n - 1))
    head = b">s" if (L + digits) % 2 == 0 else b">se"  # records at every alignment
    head_len = len(head) + digits + 1
    text = torch.empty((n, head_len + L + 1), dtype=torch.uint8, device=DEV)
    for k, c in enumerate(head):
        text[:, k] = c
    i = torch.arange(n, device=DEV)
    for d in range(digits):
        text[:, len(head) + d] = (i // 10 ** (digits - 1 - d) % 10 + 48).to(torch.uint8)
    text[:, head_len - 1] = 10
    text[:, head_len:head_len + L] = x
    text[:, head_len + L] = 10
    return text.view(-1)


class _File:
    """A file of these bytes, held in memory; `path` names it within this process."""

    def __init__(self, data):
        self.fd = os.memfd_create("case")
        view = memoryview(data)
        done = 0
        while done < len(view):
            done += os.write(self.fd, view[done:done + (1 << 30)])
        self.path = "/proc/self/fd/%d" % self.fd

    def __del__(self):
        os.close(self.fd)


def _text_of(t):
    return bytes(t.cpu().numpy()).decode()


_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = abi.Context()
    return _ctx


def _alignment(x):
    f = _fasta(x)
    torch.cuda.synchronize()
    return _context().alignment_from_fasta(f.data_ptr(), f.numel(), on_device=True)


def _np_dtype(b):
    return {1: np.uint8, 2: np.uint16, 4: np.uint32}[b]


def _torch_out(entries, b):
    return torch.zeros(max(entries, 1), device=DEV,
                       dtype={1: torch.uint8, 2: torch.int16, 4: torch.int32}[b])


def _batch_sizes(case):
    rng = np.random.default_rng(case["jobs"] * 1000 + case["n_hi"])
    n = np.exp(rng.uniform(np.log(case["n_lo"]), np.log(case["n_hi"]), case["jobs"]))
    return [(int(round(v)), int(rng.choice([1000, 5000, 10000, 29903])), int(rng.choice([1, 2])))
            for v in n]


def _distances_of(case, seed):
    """A lower triangle's values as an earlier run left them: few near zero, some large."""
    n = case["n"]
    g = _gen(seed)
    e = n * (n - 1) // 2
    v = torch.empty(e, device=DEV).exponential_(1.0 / case["mean"], generator=g)
    return v.clamp_(max=255 if case["bytes"] == 1 else 65535).to(torch.int32)


def _decimal_text(v, sep, last):
    """Decimal text of the values v with `sep` after each, and a newline
    instead after those at the positions `last`."""
    digits = torch.ones_like(v)
    for top in (10, 100, 1000, 10000):
        digits += v >= top
    size = digits + len(sep)
    size[last] = digits[last] + 1
    at = torch.cumsum(size, 0) - size
    text = torch.empty(int(size.sum()), dtype=torch.uint8, device=DEV)
    for k, c in enumerate(sep):
        on = torch.ones_like(v, dtype=torch.bool)
        on[last] = False
        text[(at + digits + k)[on]] = c
    text[(at + digits)[last]] = 10
    for k in range(5):
        on = digits > k
        text[(at + digits - 1 - k)[on]] = (v[on] // 10 ** k % 10 + 48).to(torch.uint8)
    return text.cpu().numpy()


def _lt_text(v, n):
    """Lower-triangular text (rows of comma-separated values)."""
    i = torch.arange(1, n, device=DEV)
    return _decimal_text(v, b",", i * (i + 1) // 2 - 1)


def _csv_text(v, n):
    """Full-matrix text with ", " between entries."""
    m = torch.zeros((n, n), dtype=v.dtype, device=DEV)
    i, j = torch.tril_indices(n, n, -1, device=DEV)
    m[i, j] = v
    m[j, i] = v
    return _decimal_text(m.view(-1), b", ", torch.arange(1, n + 1, device=DEV) * n - 1)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "distance":
        g = _gen(seed)
        x = _rows(2, case["L"], case["p"], g, _root(case["L"], g))
        s["pair"] = [_text_of(r) for r in x]
    elif kind == "strings":
        x, _ = _records(case, seed)
        s["list"] = [_text_of(r) for r in x]
    elif kind == "file":
        x, root = _records(case, seed)
        s["file"] = _File(_fasta(x).cpu().numpy())
        s["root"] = _text_of(root)
    elif kind == "device":
        x, root = _records(case, seed)
        s["fasta"], s["root"] = _fasta(x), _text_of(root)
        n = case["n"]
        s["out"] = _torch_out(n * (n - 1) // 2, 2 if case["wide"] else 1)
    elif kind == "resident":
        x, _ = _records(case, seed)
        s["aln"] = _alignment(x)
        n = case["n"]
        s["out"] = _torch_out(n * (n - 1) // 2, case["bytes"])
    elif kind == "batch":
        s["batch"] = _context().batch()
        s["alns"], s["outs"] = [], []
        for k, (n, L, b) in enumerate(_batch_sizes(case)):
            x, _ = _records({"n": n, "L": L, "p": case["p"]}, seed * 100 + k)
            a, o = _alignment(x), _torch_out(n * (n - 1) // 2, b)
            s["alns"].append(a)
            s["outs"].append(o)
            s["batch"].add(a, _np_dtype(b), 255 if b == 1 else 65535, o.data_ptr(), True)
    elif kind == "query":
        x, root = _records(case, seed)
        s["aln"] = _alignment(x)
        s["query"] = _text_of(_rows(1, case["L"], 5e-3, _gen(seed + 7), root)[0])
    elif kind == "text":
        v = _distances_of(case, seed)
        s["lt"] = v.to({1: torch.uint8, 2: torch.int16, 4: torch.int32}[case["bytes"]])
        room = v.numel() * (4 if case["bytes"] == 1 else 6)
        s["text"] = torch.zeros(room, dtype=torch.uint8, device=DEV)
    elif kind == "read":
        v = _distances_of(case, seed)
        s["file"] = _File((_csv_text if case["csv"] else _lt_text)(v, case["n"]))
    return s


def _bits(a):
    """uint16 values as int16 of the same bits (torch indexes no uint16)."""
    return a.view(np.int16) if a.dtype == np.uint16 else a


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "distance":
        return hd.distance(s["pair"][0], s["pair"][1])
    if kind == "strings":
        return hd.from_stringlist(s["list"]).lt_array
    if kind == "file":
        call = hd.from_fasta_large if case["wide"] else hd.from_fasta
        d = call(s["file"].path, include_x=case["include_x"], remove_duplicates=case["dup"] > 0,
                 use_gpu=case["use_gpu"])
        out = {"lt": _bits(d.lt_array)}
        if case["refs"]:
            out["refs"] = hd.fasta_reference_distances(s["root"], s["file"].path,
                                                       include_x=case["include_x"])
        return out
    if kind == "device":
        o = s["out"]
        r = hd.from_fasta_device(s["fasta"].data_ptr(), s["fasta"].numel(), o.data_ptr(),
                                 o.numel() * o.element_size(), remove_duplicates=case["dup"] > 0,
                                 max_distance=65535 if case["wide"] else 255, large=case["wide"],
                                 reference_sequence=s["root"])
        n = r["nsamples"]
        return {"lt": o[:n * (n - 1) // 2], "indices": r["sequence_indices"],
                "refs": r["reference_distances"]}
    if kind == "resident":
        top = {1: 255, 2: 65535, 4: 1 << 30}[case["bytes"]]
        _context().pairwise_lt(s["aln"], _np_dtype(case["bytes"]), top, s["out"].data_ptr(), True)
        return s["out"]
    if kind == "batch":
        s["batch"].run()
        return s["outs"]
    if kind == "query":
        return _context().alignment_reference_distances(s["aln"], s["query"])
    if kind == "text":
        nb = _context().lower_triangular_text_noalloc(s["lt"].data_ptr(), case["n"],
                                                      _np_dtype(case["bytes"]),
                                                      s["text"].data_ptr(), s["text"].numel())
        return {"text": s["text"], "bytes": nb}  # the room past the text stays zero
    if case["csv"]:
        return hd.from_csv(s["file"].path).lt_array
    call = hd.from_lower_triangular_large if case["bytes"] == 2 else hd.from_lower_triangular
    return _bits(call(s["file"].path).lt_array)


# ------------------------------------------------------------- what it takes
def work(case):
    """Bytes in and out, and the operations of the matches as a bilinear form:
    four multiply-adds for each site of each pair of distinct rows."""
    kind = case["kind"]

    def pairs(n):
        return n * (n - 1) // 2

    if kind == "distance":
        return {"bytes": 2 * case["L"] + 4, "flops": 8 * case["L"]}
    if kind == "strings":
        n, L = case["n"], case["L"]
        return {"bytes": n * L + pairs(n), "flops": 8 * pairs(n) * L}
    if kind in ("file", "device"):
        n, L = case["n"], case["L"]
        m = n - int(n * case["dup"])
        return {"bytes": n * (L + 8) + pairs(m) * (2 if case["wide"] else 1),
                "flops": 8 * pairs(m) * L}
    if kind == "resident":
        n, L = case["n"], case["L"]
        return {"bytes": n * L // 2 + pairs(n) * case["bytes"], "flops": 8 * pairs(n) * L}
    if kind == "batch":
        sizes = _batch_sizes(case)
        return {"bytes": sum(n * L // 2 + pairs(n) * b for n, L, b in sizes),
                "flops": sum(8 * pairs(n) * L for n, L, b in sizes)}
    if kind == "query":
        n, L = case["n"], case["L"]
        return {"bytes": n * L // 2 + L + 4 * n, "flops": 8 * n * L}
    # text of about two digits and a separator per entry (twice for a full matrix)
    e = pairs(case["n"])
    per = 3 * (2.3 if case.get("csv") else 1)
    return {"bytes": int(e * (case["bytes"] + per)), "flops": 0}


# ------------------------------------------------------------ exact results
def _matches(x, y, symbols, dash_with, block=1024):
    """Matching sites of every row of x with every row of y in 64 bits: equal
    symbols match, and '-' matches itself and the symbols in `dash_with`."""
    total = torch.zeros((x.shape[0], y.shape[0]), dtype=torch.float64, device=DEV)
    for c in range(0, x.shape[1], block):
        a, b = x[:, c:c + block], y[:, c:c + block]
        da, db = (a == 45), (b == 45)
        known_a, known_b = torch.zeros_like(da), torch.zeros_like(db)
        for v in symbols:
            ea, eb = (a == v), (b == v)
            known_a, known_b = known_a | ea, known_b | eb
            total += ea.double() @ eb.double().T
        if dash_with == "all":  # '-' matches every byte; other bytes are one class
            oa, ob = ~(known_a | da), ~(known_b | db)
            total += oa.double() @ ob.double().T
            known_a, known_b = ~da, ~db
        total += da.double() @ known_b.double().T + known_a.double() @ db.double().T
        total += da.double() @ db.double().T
    return total


def _triangle(x, use_gpu, include_x, top):
    n, L = x.shape
    sparse = False
    if not use_gpu:
        sparse = include_x
        if not sparse:
            same = sum(int(torch.stack([(x[:, c:c + 4096] == v).sum(0) for v in b"ACGT"]).amax(0).sum())
                       for c in range(0, L, 4096))
            sparse = (n * L - same) / (n * L) < 0.005
    symbols = b"ACGTX" if include_x else b"ACGT"
    m = _matches(x, x, symbols, "all" if sparse else "symbols")
    i, j = torch.tril_indices(n, n, -1, device=DEV)
    return (L - m[i, j]).clamp_(max=top)


def exact(case, seed):
    kind = case["kind"]
    if kind == "distance":
        g = _gen(seed)
        x = _rows(2, case["L"], case["p"], g, _root(case["L"], g))
        return case["L"] - float(_matches(x[:1], x[1:], b"ACGT", "symbols")[0, 0])
    if kind == "query":
        if case["n"] > 20000:
            return None
        x, root = _records(case, seed)
        q = _rows(1, case["L"], 5e-3, _gen(seed + 7), root)
        return case["L"] - _matches(x, q, b"ACGT", "symbols")[:, 0]
    if kind == "read":
        return None if case["csv"] else _distances_of(case, seed).double()
    if kind not in ("strings", "file", "resident") or case["n"] ** 2 * case["L"] > 4e11:
        return None
    x, root = _records(case, seed)
    if kind == "strings":
        return _triangle(x, False, False, 255)
    if kind == "resident":
        return _triangle(x, True, False, {1: 255, 2: 65535, 4: 1 << 30}[case["bytes"]])
    # duplicates leave the result: each row's first occurrence stays
    uniq = x
    if case["dup"] > 0:
        seen, keep = set(), []
        for k, r in enumerate(x.cpu().numpy()):
            b = r.tobytes()
            if b not in seen:
                seen.add(b)
                keep.append(k)
        uniq = x[torch.tensor(keep, device=DEV)]
    out = {"lt": _triangle(uniq, case["use_gpu"], case["include_x"], 65535 if case["wide"] else 255)}
    if case["refs"]:
        out["refs"] = None
    return out
