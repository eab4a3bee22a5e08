"""write_unitigs at the edges of its kernels: lines around the chars a lane
keeps as codes (28 after the k-mer), lines of 65,536 members and more (copied
by the whole grid), vertex counts around a tile of 1024 heads, and lines that
begin at every byte offset.  The lines equal the oracle's, byte for byte."""
import numpy as np
import pytest
import torch

from tests.cases import cyclic_kmers, random_seq, shuffled, text_of, walk_kmers
from unitigcoarsening_b200 import api

pytestmark = pytest.mark.gpu


def check(comp, oracle, kmers, k, method):
    text = text_of(kmers)
    d = torch.frombuffer(bytearray(text), dtype=torch.uint8).cuda()
    keys = comp.load_kmers(d, k)
    succ, pred = comp.assemble_pruned_graph(keys, k, min(8, k - 1))
    head, rank, cyc = comp.coarsen_de_bruijn_full_cycle(keys, succ, pred, k, method)
    out = comp.write_unitigs(keys, succ, head, rank, k)
    words = oracle.parse(text, k)
    osucc, opred = oracle.edges(words, k)
    ohead, orank = oracle.contract(words, k, osucc, opred)[:2]
    assert np.array_equal(api.as_u32(head), ohead) and np.array_equal(api.as_u32(rank), orank)
    assert out.cpu().numpy().tobytes() == oracle.emit(words, k, osucc, ohead, orank)


@pytest.mark.parametrize("method", [api.CONTRACT_POINTER_JUMP, api.CONTRACT_HEC])
@pytest.mark.parametrize("k", [5, 21, 31, 32, 63])
def test_line_lengths(comp, oracle, k, method):
    lens = [k + t for t in range(0, 34) for _ in range(12)] + [k + 500, k + 1, 20_000]
    kmers = []
    if k == 5:
        kmers = sorted(set(walk_kmers(random_seq(700, 3), k)))
    else:
        for i, m in enumerate(lens):
            kmers += walk_kmers(random_seq(m, 77 * k + i), k)
        kmers += cyclic_kmers(90, k, seed=6)
    check(comp, oracle, shuffled(kmers, 2), k, method)


@pytest.mark.parametrize("method", [api.CONTRACT_POINTER_JUMP, api.CONTRACT_HEC])
@pytest.mark.parametrize("k", [31, 63])
def test_huge_lines(comp, oracle, k, method):
    kmers = []
    for i, m in enumerate([65_535, 65_536, 65_537, 200_000, 1, 3]):
        kmers += walk_kmers(random_seq(m + k - 1, 9 * k + i), k)
    check(comp, oracle, shuffled(kmers, 8), k, method)


@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 1025, 4099])
def test_tile_edges(comp, oracle, n):
    k = 31
    check(comp, oracle, walk_kmers(random_seq(n + k - 1, n), k)[::-1], k, api.CONTRACT_POINTER_JUMP)
    iso = [random_seq(k, 10_000 + i) for i in range(n)]
    check(comp, oracle, iso, k, api.CONTRACT_HEC)


@pytest.mark.parametrize("n", [3, 1023, 1027, 5000])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_head_array_at_any_word(comp, oracle, n, shift):
    """head and rank may start at any word of a larger array."""
    k = 31
    kmers = walk_kmers(random_seq(n // 2 + k - 1, n), k)[::-1] + [random_seq(k, 500 + i) for i in range(n - n // 2)]
    text = text_of(shuffled(kmers, 4))
    keys = comp.load_kmers(torch.frombuffer(bytearray(text), dtype=torch.uint8).cuda(), k)
    succ, pred = comp.assemble_pruned_graph(keys, k, 8)
    head, rank, _ = comp.coarsen_de_bruijn_full_cycle(keys, succ, pred, k)
    want = comp.write_unitigs(keys, succ, head, rank, k).cpu().numpy().tobytes()
    words = oracle.parse(text, k)
    osucc, opred = oracle.edges(words, k)
    assert want == oracle.emit(words, k, osucc, *oracle.contract(words, k, osucc, opred)[:2])
    moved = []
    for t in (head, rank):
        buf = torch.empty(n + shift, dtype=t.dtype, device=t.device)
        buf[shift:] = t
        moved.append(buf[shift:])
    assert comp.write_unitigs(keys, succ, *moved, k).cpu().numpy().tobytes() == want
