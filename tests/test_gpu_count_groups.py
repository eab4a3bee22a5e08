"""The scatter's third level where the pack counts groups of buckets (2^24
buckets and more), so that it counts each bucket itself: sub-partitions that are
empty, of a few records, past what a block holds in registers (4096, and 2560
with two key words) and past its staging (8192 and 4096), one and two key
words.  Lines equal the oracle's."""
import random

import pytest
import torch

from tests.cases import random_seq, shuffled, sorted_lines, text_of, walk_kmers

pytestmark = pytest.mark.gpu


def with_cores(k, sizes, seed):
    """k-mers around 16-char cores, sizes[i] around the i-th: where a core holds
    the minimizer they share a bucket."""
    r = random.Random(seed)
    out = set()
    for n in sizes:
        core = "".join(r.choices("ACGT", k=16))
        for _ in range(n):
            x = "".join(r.choices("ACGT", k=k - 16))
            i = r.randrange(k - 15)
            out.add(x[:i] + core + x[i:])
    return sorted(out)


@pytest.mark.parametrize("k", [31, 47])
@pytest.mark.parametrize("bits", [24, 25])
@pytest.mark.parametrize("kind", ["few", "walk", "cores"])
def test_count_groups(comp, oracle, k, bits, kind):
    if kind == "few":
        kmers = walk_kmers(random_seq(k + 99, 5), k)
    elif kind == "walk":
        kmers = walk_kmers(random_seq(300_000, k + bits), k)
    else:
        kmers = with_cores(k, [3000, 5000, 9000, 20_000, 50_000] * 4, 7 * k + bits)
    text = text_of(shuffled(kmers, 1))
    want = sorted_lines(oracle.compact(text, k)[0])
    dev = torch.frombuffer(bytearray(text), dtype=torch.uint8).cuda()
    comp.set_tuning(bucket_bits=bits)
    try:
        got, st = comp.compact(dev, k, 8, stats=True)
        assert st["bucket_bits"] == bits
        assert kind != "cores" or st["n_big_tiles"] > 0
        assert sorted_lines(got.cpu().numpy().tobytes()) == want
        comp.set_sorted_output(True)
        got = comp.compact(dev, k, 8)
        assert got.cpu().numpy().tobytes() == b"".join(x + b"\n" for x in want)
    finally:
        comp.set_sorted_output(False)
        comp.set_tuning(bucket_bits=0)
