"""Pointer-jumping contraction over chains of chosen lengths: lines shorter
and longer than a vertex's first walk, lengths around its end, cycles, and
vertex counts around the blocks that work them, against a direct walk of the
chains."""
import ctypes

import numpy as np
import pytest
import torch

from unitigcoarsening_b200 import api

pytestmark = pytest.mark.gpu


def graph(lengths, cycles, seed):
    """Chains and cycles of those lengths over shuffled ids: succ, pred and
    the expected head and rank (a cycle starts at its smallest key; the keys
    here are the ids)."""
    n = sum(lengths) + sum(cycles)
    ids = np.random.default_rng(seed).permutation(n).astype(np.int64)
    succ, pred = np.full(n, -1, np.int32), np.full(n, -1, np.int32)
    head, rank = np.empty(n, np.int32), np.empty(n, np.int32)
    at = 0
    for i, m in enumerate(list(lengths) + list(cycles)):
        c = ids[at: at + m]
        at += m
        succ[c[:-1]], pred[c[1:]] = c[1:], c[:-1]
        if i >= len(lengths):
            succ[c[-1]], pred[c[0]] = c[0], c[-1]
            c = np.roll(c, -int(np.argmin(c)))
        head[c], rank[c] = c[0], np.arange(m)
    return n, succ, pred, head, rank


@pytest.mark.parametrize("lengths,cycles", [
    ([1], []),
    ([8], []),
    ([9], []),
    (list(range(1, 41)), []),
    ([7, 8, 9, 10] * 64 + [16, 17, 18, 33, 65] * 8, []),
    ([1023], []),
    ([1024], []),
    ([1025, 1], []),
    ([2] * 2000 + [5000, 1, 12345, 100_000], []),
    ([1] * 300_000 + [2] * 100_000 + [31] * 1000, []),
    ([3, 9], [1, 2, 8, 9, 300]),
    ([50_000], [4000]),
])
def test_contract_chains(comp, lengths, cycles):
    n, succ, pred, head, rank = graph(lengths, cycles, 11 + len(lengths))
    keys = torch.arange(n, dtype=torch.int64, device="cuda").view(-1, 1)
    h, r, nc = comp.coarsen_de_bruijn_full_cycle(
        keys, torch.from_numpy(succ).cuda(), torch.from_numpy(pred).cuda(), 31)
    assert nc == len(cycles)
    np.testing.assert_array_equal(h.cpu().numpy(), head)
    np.testing.assert_array_equal(r.cpu().numpy(), rank)


def test_contract_in_place(comp):
    """Results may overwrite the predecessors."""
    n, succ, pred, head, rank = graph([1, 9, 400, 77], [], 5)
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
