"""Site lists of more tiles of rows than one launch's grid holds: the build takes
them in several launches, and the sites whose reference matches nothing count
once. Row ranges at the end of such an alignment against the sites' own rule."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE, SLICE = 224, 65535  # rows of a tile, tiles of a launch


def test_zero_sites_count_once(monkeypatch):
    torch = pytest.importorskip("torch")
    from hammingdist_gb300 import abi

    n, L = TILE * SLICE + 300, 8
    free, _ = torch.cuda.mem_get_info()
    if free < 24 << 30:
        pytest.skip("needs 24 GB of device memory")
    # every row "NNACGTAC" but for one site of every 7th row
    text = torch.empty((n, L + 3), dtype=torch.uint8, device="cuda")
    text[:] = torch.tensor(list(b">\nNNACGTAC\n"), dtype=torch.uint8, device="cuda")
    text[::7, 2 + 4] = ord("T")
    torch.cuda.synchronize()
    monkeypatch.setenv("HAMMINGDIST_SITE_LISTS", "1")
    ctx = abi.Context(0)
    try:
        aln = ctx.alignment_from_fasta(text.data_ptr(), text.numel(), on_device=True)
        del text
        # the last tile row of 128: its rows against all earlier ones
        lo = (n - 1) // 128 * 128
        base = lo * (lo - 1) // 2
        out = torch.empty(n * (n - 1) // 2 - base, dtype=torch.uint8, device="cuda")
        fn = getattr(abi.lib(), "_ZN2hd14pairwise_tilesEP6hd_ctxPK12hd_alignmentijPvmjj")
        fn.restype = None
        fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_uint32,
                       ctypes.c_void_p, ctypes.c_uint64, ctypes.c_uint32, ctypes.c_uint32]
        fn(ctx.h, aln.h, 1, 255, out.data_ptr(), base, lo // 128, lo // 128 + 1)
        ctx.synchronize()
        odd = torch.arange(n, device="cuda") % 7 == 0
        at = 0
        for i in range(lo, n):  # N matches nothing: two sites, and the substituted one
            want = 2 + (odd[:i] != odd[i]).to(torch.uint8)
            assert torch.equal(out[at:at + i], want), i
            at += i
        aln.free()
    finally:
        ctx.close()
