"""from_lower_triangular's flat reader around its tiles: fields across tile
edges, of every shape std::stoi takes, and the first error in file order."""
import numpy as np
import pytest

from gpu_util import write
from oracle import hd_formats as fm

pytestmark = pytest.mark.gpu
hd = pytest.importorskip("hammingdist_gb300")


def _lines(rng, n, kinds):
    out = []
    for i in range(1, n):
        row = []
        for _ in range(i):
            k = rng.choice(kinds)
            v = int(rng.integers(0, 10 ** int(rng.integers(1, 6))))
            row.append({"plain": "%d", "space": "  %d", "sign": "+%d", "zeros": "0000000%d",
                        "trail": "%d x", "cr": "%d\r"}[k] % v)
        out.append(",".join(row))
    return out


@pytest.mark.parametrize("kinds", [["plain"], ["plain", "space", "sign", "zeros", "trail", "cr"]])
@pytest.mark.parametrize("end", ["\n", "", "\r\n"])
@pytest.mark.parametrize("n", [2, 40, 130, 260])
def test_read_fields(tmp_path, kinds, end, n):
    text = ("\n".join(_lines(np.random.default_rng(n), n, kinds)) + end).encode()
    path = write(tmp_path, "a.txt", text)
    for call, dtype in ((hd.from_lower_triangular, np.uint8),
                        (hd.from_lower_triangular_large, np.uint16)):
        want = fm.from_lower_triangular(text, dtype)[0]
        np.testing.assert_array_equal(np.asarray(call(path).lt_array), want)


@pytest.mark.parametrize("where", [0, 4090, 4095, 4096, 8191, 20000])
@pytest.mark.parametrize("bad,error", [(b"x", ValueError), (b"", ValueError),
                                       (b"99999999999", IndexError)])
def test_read_errors_across_tiles(tmp_path, where, bad, error):
    # the first bad field decides, wherever the tiles' edges fall
    fields = [b"12"] * 9000
    k = where // 3
    fields[k] = bad
    fields[-1] = b"y" if error is IndexError else b"99999999999"
    path = write(tmp_path, "b.txt", b",".join(fields) + b"\n")
    with pytest.raises(error):
        hd.from_lower_triangular(path)


def test_read_ends_with_a_comma(tmp_path):
    with pytest.raises(ValueError):
        hd.from_lower_triangular(write(tmp_path, "c.txt", b"1\n2,3,"))
