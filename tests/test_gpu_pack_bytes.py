"""Text to keys where many bytes of a line are not ACGT: any of them, in any
number, at any place, and a line break among them; and the time of it."""
import random
import statistics
import time

import numpy as np
import pytest
import torch

from unitigcoarsening_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [2, 15, 21, 31, 32, 33, 47, 63])
@pytest.mark.parametrize("share", [0.1, 0.6, 1.0])
@pytest.mark.parametrize("column", ["", "\t3"])
def test_many_other_bytes(comp, oracle, k, share, column):
    r = random.Random(k)
    other = [b for b in range(256) if b not in b"ACGT\n"]
    near = [0x08, 0x0C, 0x0E, 0x1A, 0x0B, 0x4A, 0x61, 0x63, 0x67, 0x74, 0x45, 0x50, 0x51, 0xC1, 0x8A]
    rows = [bytes(r.choice(near if r.random() < 0.5 else other) if r.random() < share else r.choice(b"ACGT")
                  for _ in range(k)) for _ in range(1300)]
    text = b"1300\n" + b"".join(x + column.encode() + b"\n" for x in rows)
    dev = torch.frombuffer(bytearray(text), dtype=torch.uint8).cuda()
    got = api.keys_to_words(comp.load_kmers(dev, k), k)
    assert np.array_equal(got.reshape(-1), np.asarray(oracle.parse(text, k)).reshape(-1))
    if not column:  # a line cut short among such bytes, the total size as before
        bad = bytearray(text)
        bad[5 + 700 * (k + 1) + k] = ord("x")
        bad[5 + 700 * (k + 1) + k // 2] = ord("\n")
        with pytest.raises(api.UCError):
            comp.load_kmers(torch.frombuffer(bad, dtype=torch.uint8).cuda(), k)


def test_other_bytes_are_not_slow(comp):
    """A text without one letter of ACGT packs in twice the time of a regular one
    (2.6 times when each such byte was cleared by itself)."""
    km = synth.kmer_set(synth.GenomeSpec(length=5_000_000, gc=0.5, seed=1), 31, "cuda")
    t = []
    for lower in (False, True):
        lines = synth.kmers_to_lines(km, 31)
        if lower:
            lines[:, :31] += 32
        head = torch.tensor(list(f"{km.shape[0]}\n".encode()), dtype=torch.uint8, device="cuda")
        text = torch.cat([head, lines.flatten()])
        v = []
        for _ in range(20):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            comp.load_kmers(text, 31)
            torch.cuda.synchronize()
            v.append(time.perf_counter() - t0)
        t.append(statistics.median(v[5:]))
    assert t[1] < 2 * t[0], t
