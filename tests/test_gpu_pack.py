"""Text to keys at the edges of the pack's passes (512 lines, 16-byte pieces):
widths around one piece per line, line counts around a pass, every offset of
the first line, every byte value among a line's chars, and a wrong byte in a
line break's place.  Keys equal the oracle's parse, bit for bit."""
import random

import numpy as np
import pytest
import torch

from unitigcoarsening_b200 import api

pytestmark = pytest.mark.gpu


def dev(b: bytes):
    return torch.frombuffer(bytearray(b), dtype=torch.uint8).cuda()


def keys_equal(comp, oracle, text: bytes, k: int):
    got = api.keys_to_words(comp.load_kmers(dev(text), k), k)
    want = oracle.parse(text, k)
    assert np.array_equal(got.reshape(-1), np.asarray(want).reshape(-1))


def lines(n: int, k: int, seed: int):
    r = random.Random(seed)
    return ["".join(r.choices("ACGT", k=k)) for _ in range(n)]


@pytest.mark.parametrize("k", [2, 14, 15, 16, 21, 31, 32, 47, 63])
@pytest.mark.parametrize("n", [1, 511, 512, 513, 1025, 2600])
def test_line_counts_and_first_line_offsets(comp, oracle, k, n):
    body = "\n".join(lines(n, k, n + k)) + "\n"
    for pad in range(0, 16, 1 if n == 513 else 7):
        keys_equal(comp, oracle, (" " * pad + f"{n}\n" + body).encode(), k)


@pytest.mark.parametrize("k", [14, 21, 31, 63])
@pytest.mark.parametrize("column", ["", "\t17"])
def test_every_byte_value(comp, oracle, k, column):
    """Bytes that are not ACGT pack as A, wherever they stand in a line."""
    r = random.Random(k)
    rows = [bytearray(x.encode()) for x in lines(3000, k, 5)]
    values = [b for b in range(256) if b != 0x0A]
    for i, b in enumerate(values * 8):
        rows[7 * i % 3000][r.randrange(k)] = b
    text = b"3000\n" + b"".join(bytes(x) + column.encode() + b"\n" for x in rows)
    keys_equal(comp, oracle, text, k)


@pytest.mark.parametrize("k", [14, 15, 31, 63])
@pytest.mark.parametrize("byte", [0x08, 0x0E, 0x1D, 0x0D, 0x41, 0x43, 0x00])
def test_wrong_byte_in_a_break_is_an_error(comp, k, byte):
    """Two lines run together: the count no longer matches."""
    text = bytearray(("1500\n" + "\n".join(lines(1500, k, 3)) + "\n").encode())
    text[5 + 700 * (k + 1) + k] = byte
    with pytest.raises(api.UCError) as e:
        comp.load_kmers(dev(bytes(text)), k)
    assert e.value.status == 1


@pytest.mark.parametrize("k", [15, 31, 63])
def test_break_inside_a_line_is_an_error(comp, k):
    """A line cut short by a break, the total size as for full lines."""
    text = bytearray(("1500\n" + "\n".join(lines(1500, k, 4)) + "\n").encode())
    text[5 + 700 * (k + 1) + k] = ord("A")
    text[5 + 700 * (k + 1) + 3] = ord("\n")
    with pytest.raises(api.UCError) as e:
        comp.load_kmers(dev(bytes(text)), k)
    assert e.value.status == 1


@pytest.mark.parametrize("k", [5, 21, 63])
@pytest.mark.parametrize("n", [1, 2, 500, 9000])
@pytest.mark.parametrize("end", ["\n", "", "\r\n\n\n"])
def test_line_index(comp, oracle, k, n, end):
    """Lines of different widths (columns after the k-mer), among them one
    wider than a chunk of the index and breaks on both sides of its edges."""
    r = random.Random(n * k)
    rows = [x + "\t" + "7" * r.randrange(0, 40) for x in lines(n, k, n)]
    rows[n // 2] += "9" * 40_000
    for pad in (0, 5, 11):
        keys_equal(comp, oracle, (" " * pad + f"{n}\n" + "\n".join(rows) + end).encode(), k)
    with pytest.raises(api.UCError):
        comp.load_kmers(dev((f"{n + 1}\n" + "\n".join(rows) + end).encode()), k)
