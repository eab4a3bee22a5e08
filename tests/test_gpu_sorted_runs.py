"""Sorted output where many lines begin with the same chars: bins of more
lines than a few tiles hold are sorted by the whole grid.  Sizes around the
limit (five windows of 250, 500 or 1000 lines), around its chunks of 4096
records, several such bins at once, prefixes that leave one digit or all of
them to sort by, one and two key words, lines as records, as text and long
ones.  Lines equal the oracle's byte for byte."""
import random
import statistics
import time

import pytest
import torch

from tests.cases import random_seq, shuffled, sorted_lines, text_of, walk_kmers

pytestmark = pytest.mark.gpu


def sharing(n, k, shared, seed):
    """n distinct k-mers with one random prefix of `shared` chars."""
    r = random.Random(seed)
    pre = "".join(r.choices("ACGT", k=shared))
    tails = set()
    while len(tails) < n:
        tails.add("".join(r.choices("ACGT", k=k - shared)))
    return [pre + x for x in sorted(tails)]


def others(n, k, seed):
    r = random.Random(seed)
    return ["".join(r.choices("ACGT", k=k)) for _ in range(n)]


def check(comp, oracle, kmers, k, shift=3):
    text = text_of(shuffled(sorted(set(kmers)), 11))
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
    assert bool((buf[shift + m:] == 0x55).all())


@pytest.mark.parametrize("k,shared", [(31, 12), (31, 20), (32, 14), (33, 20), (63, 12), (63, 45)])
@pytest.mark.parametrize("n", [1249, 1252, 2502, 4095, 4097, 8192, 20_001])
def test_one_bin(comp, oracle, k, shared, n):
    check(comp, oracle, sharing(n, k, shared, 10 * k + n) + others(2000, k, n), k)


@pytest.mark.parametrize("k", [15, 31, 63])
@pytest.mark.parametrize("rest", [0, 400_000])
def test_several_bins(comp, oracle, k, rest):
    """Bins of many sizes, next to each other and apart, first and last."""
    kmers = others(rest, k, 5)
    for i, (n, pre) in enumerate([(6000, "A" * 10), (3000, "AAAAAAAAAC"), (5100, "AAAAAAAAAG"), (12_289, "C" * 9),
                                  (1300, "GTACGATC"), (70_000 if k > 15 else 4000, "GTACGATG"), (5500, "T" * 8)]):
        kmers += [pre + x for x in others(n, k - len(pre), 100 + i)]
    check(comp, oracle, kmers, k, shift=9)


@pytest.mark.parametrize("k", [21, 31, 47])
@pytest.mark.parametrize("warp_capacity", [0, 1])
def test_line_lengths_in_a_bin(comp, oracle, k, warp_capacity):
    """Paths of all kinds that begin with the same chars; warp_capacity 1:
    every line reaches the sort as text."""
    kmers, pre = [], "ACCATAGGACA"
    for i, m in enumerate([k, k + 1, k + 5, k + 28, k + 29, k + 40, 300] * 400 + [70_000]):
        kmers += walk_kmers(pre + random_seq(m - len(pre), 7000 * k + i), k)
    comp.set_tuning(warp_capacity=warp_capacity)
    try:
        check(comp, oracle, kmers + sharing(9000, k, 11, 3), k)
    finally:
        comp.set_tuning(warp_capacity=0)


@pytest.mark.parametrize("k", [31, 63])
def test_a_hundred_bins(comp, oracle, k):
    kmers = []
    for i in range(100):
        pre = "".join("ACGT"[(i * 41 >> (2 * j)) & 3] for j in range(6)) + "GAT"
        kmers += [pre + x for x in others(1251 + i, k - len(pre), 700 + i)]
    check(comp, oracle, kmers + others(500, k, 1), k)


@pytest.mark.parametrize("k", [31, 63])
@pytest.mark.parametrize("bins,n", [(1200, 5200), (3, 1_500_000)])
def test_millions_of_lines_in_bins(comp, k, bins, n):
    """Unrelated k-mers, so every line is one of them: the text sorted."""
    from unitigcoarsening_b200 import synth
    v = torch.arange(bins * n, device="cuda")
    w = synth._srl(synth.rand_u64(9, 3, v), 64 - 2 * 31)
    w = (w & ((1 << 38) - 1)) | ((v // n * 7919 + 3) << 38)
    if k == 63:
        w = torch.stack([((w << 2) | (v & 3)) ^ (-(1 << 63)), synth._srl(synth.rand_u64(9, 4, v), 64 - 2 * 31)], 1)
        w = synth._unique_rows(w)
    else:
        w = torch.unique(w)
    text = synth.format_text(synth.shuffle(w, 1), k)
    comp.set_sorted_output(True)
    try:
        got = comp.compact(text, k, 8)
    finally:
        comp.set_sorted_output(False)
    assert torch.equal(got, synth.kmers_to_lines(w, k).flatten())


def test_shared_prefix_is_not_slow(comp):
    """300,000 lines with one prefix among a million others: ordering them costs
    at most as much as the rest of the call does twice over (it costs less than
    the rest for unrelated lines; one block sorting them took ten times the
    rest)."""
    from unitigcoarsening_b200 import synth
    k, n, m = 31, 300_000, 1_000_000
    w = synth._srl(synth.rand_u64(5, 3, torch.arange(n + m, device="cuda")), 64 - 2 * k)
    w[:n] = (w[:n] & ((1 << 38) - 1)) | (0x5A5A5A << 38)
    text = synth.format_text(synth.shuffle(torch.unique(w), 1), k)
    out = torch.empty(comp.output_bound(text.numel(), k), dtype=torch.uint8, device="cuda")
    times = []
    for ordered in (False, True):
        comp.set_sorted_output(ordered)
        try:
            t = []
            for _ in range(9):
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                comp.compact(text, k, 8, out=out)
                torch.cuda.synchronize()
                t.append(time.perf_counter() - t0)
        finally:
            comp.set_sorted_output(False)
        times.append(statistics.median(t[2:]))
    assert times[1] < 3 * times[0], times
