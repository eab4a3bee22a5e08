"""Contraction of long lines (the k-mers of one strand): from 2^19 vertices with
more than three quarters of them unranked after the walk, the rounds run over
every vertex.  Vertex counts and line lengths around both limits, cycles, in
place, and the time against that of short lines.  HEC: one line of millions of
vertices in several orders."""
import ctypes
import statistics
import time

import numpy as np
import pytest
import torch

from tests.test_gpu_contract import graph
from unitigcoarsening_b200 import api

pytestmark = pytest.mark.gpu

N0 = 1 << 19


def run(comp, n, succ, pred, method=api.CONTRACT_POINTER_JUMP):
    keys = torch.arange(n, dtype=torch.int64, device="cuda").view(-1, 1)
    return comp.coarsen_de_bruijn_full_cycle(keys, torch.from_numpy(succ).cuda(), torch.from_numpy(pred).cuda(), 31,
                                             method)


@pytest.mark.parametrize("lengths,cycles", [
    ([N0 - 1], []),
    ([N0], []),
    ([N0 + 1], []),
    ([31] * (N0 // 30), []),
    ([32] * (N0 // 31), []),
    ([33] * (N0 // 32), []),
    ([40] * 14_000, []),
    ([1000] * 700 + [1] * 130_000, []),
    ([1000] * 700 + [1] * 260_000, []),
    ([1000] * 700 + list(range(1, 200)), [1, 2, 300, 5000]),
    ([2_000_003], []),
    ([], [600_000]),
])
def test_contract_long_lines(comp, lengths, cycles):
    n, succ, pred, head, rank = graph(lengths, cycles, 3 + len(lengths))
    h, r, nc = run(comp, n, succ, pred)
    assert nc == len(cycles)
    np.testing.assert_array_equal(h.cpu().numpy(), head)
    np.testing.assert_array_equal(r.cpu().numpy(), rank)


def test_contract_long_lines_in_place(comp):
    n, succ, pred, head, rank = graph([700_000, 9], [], 5)
    keys = torch.arange(n, dtype=torch.int64, device="cuda").view(-1, 1)
    ds, dp = torch.from_numpy(succ).cuda(), torch.from_numpy(pred).cuda()
    dr = torch.empty_like(dp)
    torch.cuda.synchronize()
    nc = ctypes.c_uint64()
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert comp._L.uc_contract(comp._h, p(keys), p(ds), p(dp), n, 31, api.CONTRACT_POINTER_JUMP, p(dp), p(dr),
                               ctypes.byref(nc)) == 0
    np.testing.assert_array_equal(dp.cpu().numpy(), head)
    np.testing.assert_array_equal(dr.cpu().numpy(), rank)


def test_rounds_grow_with_the_log_of_the_length(comp):
    """Lines of 1000 take at most log(1000) / log(20) = 2.3 times as long as
    lines of 20, and a tenth more (2.9 times when every round gathered twice)."""
    n = 8_000_000
    t = []
    for m in (20, 1000):
        ids = torch.randperm(n, device="cuda", dtype=torch.int32,
                             generator=torch.Generator("cuda").manual_seed(m)).view(-1, m)
        succ = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        pred = succ.clone()
        succ[ids[:, :-1].flatten().long()] = ids[:, 1:].flatten()
        pred[ids[:, 1:].flatten().long()] = ids[:, :-1].flatten()
        keys = torch.arange(n, dtype=torch.int64, device="cuda").view(-1, 1)
        v = []
        for _ in range(12):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            comp.coarsen_de_bruijn_full_cycle(keys, succ, pred, 31)
            torch.cuda.synchronize()
            v.append(time.perf_counter() - t0)
        t.append(statistics.median(v[3:]))
    assert t[1] < 2.3 * 1.1 * t[0], t


@pytest.mark.parametrize("order", ["ascending", "descending", "shuffled", "interleaved"])
def test_hec_one_line(comp, order):
    """One line of 4M vertices: the rounds finish, with no wait running out."""
    n = 4_000_000
    ids = {"ascending": lambda: np.arange(n), "descending": lambda: np.arange(n)[::-1].copy(),
           "shuffled": lambda: np.random.default_rng(1).permutation(n),
           "interleaved": lambda: np.arange(n).reshape(-1, 2000).T.flatten().copy()}[order]()
    succ, pred = np.full(n, -1, np.int32), np.full(n, -1, np.int32)
    succ[ids[:-1]], pred[ids[1:]] = ids[1:], ids[:-1]
    comp.set_faults(hec_strict=True)
    try:
        h, r, nc = run(comp, n, succ, pred, api.CONTRACT_HEC)
    finally:
        comp.set_faults()
    assert nc == 0
    assert bool((h == int(ids[0])).all())
    np.testing.assert_array_equal(r.cpu().numpy()[ids], np.arange(n))
