"""Sorted output at the edges of its kernels: line counts around a tile's
window and capacity, lines around the chars a record holds (28 after the
k-mer) and around the length the whole grid copies (65,536 bytes), bins of
more lines than a tile sorts in shared memory, one and two key words, and
output buffers at odd bytes.  The whole output equals the oracle's lines in
byte order, byte for byte; bytes outside it stay as they were."""
import random

import pytest
import torch

from tests.cases import random_seq, shuffled, sorted_lines, text_of, walk_kmers

pytestmark = pytest.mark.gpu


def check(comp, oracle, text: bytes, k: int, shift: int = 0):
    expect = b"".join(x + b"\n" for x in sorted_lines(oracle.compact(text, k)[0]))
    d = torch.frombuffer(bytearray(text), dtype=torch.uint8).cuda()
    buf = torch.full((comp.output_bound(len(text), k) + 32,), 0x55, dtype=torch.uint8, device="cuda")
    comp.set_sorted_output(True)
    try:
        got = comp.compact(d, k, min(8, k - 1), out=buf[shift:])
    finally:
        comp.set_sorted_output(False)
    m = got.numel()
    assert got.cpu().numpy().tobytes() == expect
    assert bool((buf[:shift] == 0x55).all())
    assert bool((buf[shift + m + 64:] == 0x55).all())


@pytest.mark.parametrize("k", [31, 32, 63])
@pytest.mark.parametrize("n", [1, 2, 255, 257, 1023, 1025, 2049, 70_001])
def test_line_counts(comp, oracle, k, n):
    """n unrelated k-mers: n lines of one k-mer each."""
    r = random.Random(100 * k + n)
    kmers = ["".join(r.choices("ACGT", k=k)) for _ in range(n)]
    check(comp, oracle, text_of(kmers), k, shift=n % 16)


@pytest.mark.parametrize("k,shared,n", [(31, 12, 2049), (31, 12, 6000), (31, 20, 3000), (63, 12, 5000),
                                        (63, 40, 4099)])
def test_lines_that_share_their_first_chars(comp, oracle, k, shared, n):
    """More lines with one prefix than a tile holds, among others."""
    r = random.Random(7 * k + n)
    pre = "".join(r.choices("ACGT", k=shared))
    kmers = {pre + "".join(r.choices("ACGT", k=k - shared)) for _ in range(n)}
    kmers |= {"".join(r.choices("ACGT", k=k)) for _ in range(3000)}
    check(comp, oracle, text_of(shuffled(sorted(kmers), 3)), k, shift=5)


@pytest.mark.parametrize("k", [21, 31, 33, 63])
@pytest.mark.parametrize("lengths", ["tails", "long", "huge"])
def test_line_lengths(comp, oracle, k, lengths):
    """Paths of chosen lengths, each one line."""
    if lengths == "tails":
        lens = [k + t for t in range(0, 36) for _ in range(40)]
    elif lengths == "long":
        lens = [k, k + 1, k + 28, k + 29, 300, 1000, 16384 - k, 16384, 16500, 40_000] * 6
    else:
        lens = [k, k + 5, 65_534, 65_535, 65_536, 150_000, k + 29] * 2
    kmers = []
    for i, m in enumerate(lens):
        kmers += walk_kmers(random_seq(m, 1000 * k + i), k)
    check(comp, oracle, text_of(shuffled(kmers, 5)), k, shift=k % 7)


@pytest.mark.parametrize("k", [2, 3, 5, 8])
def test_small_k(comp, oracle, k):
    kmers = sorted(set(walk_kmers(random_seq(40 * 4 ** min(k, 5) // 10 + k, 9), k)))
    check(comp, oracle, text_of(shuffled(kmers, 1)), k, shift=1)


@pytest.mark.parametrize("k", [31, 63])
@pytest.mark.parametrize("tuning", [dict(warp_capacity=1), dict(warp_capacity=32), dict(warp_capacity=1024),
                                    dict(tile_capacity=256, bucket_fill=1), dict(load_factor_pct=150),
                                    dict(contract_method=1)])
def test_lines_from_every_tier(comp, oracle, k, tuning):
    """Lines that come as records (warp tiles), as text (block and oversized
    tiles, stitched lines) and both, with cycles among them."""
    from tests.cases import cyclic_kmers
    kmers = []
    for i, m in enumerate([k, k + 1, k + 3, k + 28, k + 29, k + 30, 400] * 300):
        kmers += walk_kmers(random_seq(m, 5000 * k + i), k)
    kmers += cyclic_kmers(k + 40, k, seed=2) + cyclic_kmers(300, k, seed=8)
    comp.set_tuning(**tuning)
    try:
        check(comp, oracle, text_of(shuffled(kmers, 4)), k, shift=9)
    finally:
        comp.set_tuning(**{f: 0 for f in tuning})
