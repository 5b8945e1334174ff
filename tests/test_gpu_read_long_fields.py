"""Lower-triangular text with long fields: what follows a number is not read, and
whitespace, signs and empty fields at the ends of lines keep std::stoi's rules."""
import time

import numpy as np
import pytest

hd = pytest.importorskip("hammingdist_gb300")

pytestmark = pytest.mark.gpu


def _read(tmp_path, text):
    p = tmp_path / "lt.txt"
    p.write_bytes(text)
    return np.array(hd.from_lower_triangular_large(str(p)).lt_array)


@pytest.mark.parametrize("tail", [b"\n", b"", b"\n1,2\n"])
def test_junk_after_a_number(tmp_path, tail):
    junk = b"7" + b"z" * (16 << 20) + tail
    want = [7, 1, 2] if len(tail) > 1 else [7]
    _read(tmp_path, b"1\n")  # the library is there
    t = time.perf_counter()
    np.testing.assert_array_equal(_read(tmp_path, junk), np.array(want, np.uint16))
    # one thread that reads to the field's end takes 0.9 s
    assert time.perf_counter() - t < 0.4


@pytest.mark.parametrize("text,want", [
    (b" 5\n\t6,\v7\n\f8 ,\r9\r,+10\n", [5, 6, 7, 8, 9, 10]),
    (b"5 x\n 12345  7,\t 65536\n", [5, 12345, 65535]),
    (b"1\n2,3" + b" " * 5000, [1, 2, 3]),
    (b"1\n" + b" " * 5000 + b"2,3", [1, 2, 3]),
    (b"70000\n1e3,0x10\n", [65535, 1, 0]),
])
def test_rules_at_the_ends(tmp_path, text, want):
    np.testing.assert_array_equal(_read(tmp_path, text), np.array(want, np.uint16))


@pytest.mark.parametrize("text", [b"1\n \n2\n", b"1\n2, \n", b"1\n2,\t", b"1\n+\n2\n", b"1\n-,2\n",
                                  b"1\n\n", b"1\n2,", b" ", b"1\n \r\n5\n", b"1\n+ 3,4\n"])
def test_fields_without_a_number(tmp_path, text):
    with pytest.raises(ValueError, match="stoi"):
        _read(tmp_path, text)
