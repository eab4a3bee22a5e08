"""The three scatter levels at the edges of their blocks: k-mer counts around a
level-1 chunk (3072, or 2048 with two key words), bucket counts that leave
sub-partitions empty, of a few records, past what a block keeps in registers
(4096 and 2560) and past its staging, with and without a second level.  The
kept edges and the lines equal the oracle's."""
import random

import numpy as np
import pytest
import torch

from unitigcoarsening_b200 import as_u32

pytestmark = pytest.mark.gpu


def text_of(n, k, seed, letters="ACGT"):
    r = random.Random(seed)
    g = "".join(r.choices(letters, k=n + k + 200))
    kmers = sorted({g[i: i + k] for i in range(len(g) - k + 1)})[:n]
    r.shuffle(kmers)
    assert len(kmers) == n
    return (f"{n}\n" + "\n".join(kmers) + "\n").encode()


@pytest.mark.parametrize("k", [31, 47])
@pytest.mark.parametrize("n,bits", [
    (1, 1), (100, 1), (2047, 3), (2048, 6), (2049, 10), (3071, 3), (3072, 9), (3073, 20),
    (20_000, 1), (20_000, 2), (20_000, 17), (60_000, 4), (60_000, 12),
])
def test_scatter_levels(comp, oracle, k, n, bits):
    text = text_of(n, k, n + bits)
    words = oracle.parse(text, k)
    osucc, opred = oracle.edges(words, k)
    ohead, orank = oracle.contract(words, k, osucc, opred)[:2]
    want = sorted(oracle.emit(words, k, osucc, ohead, orank).split(b"\n")[:-1])
    dev = torch.frombuffer(bytearray(text), dtype=torch.uint8).cuda()
    comp.set_tuning(bucket_bits=bits)
    try:
        succ, pred = comp.assemble_pruned_graph(comp.load_kmers(dev, k), k, 8)
        assert np.array_equal(as_u32(succ), osucc)
        assert np.array_equal(as_u32(pred), opred)
        got = comp.compact(dev, k, 8).cpu().numpy().tobytes()
    finally:
        comp.set_tuning(bucket_bits=0)
    assert sorted(got.split(b"\n")[:-1]) == want
