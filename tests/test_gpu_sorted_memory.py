"""Device memory of sorted output: the context's scratch stays within its
budget whatever the lines come from (warp_capacity 1: every line reaches the sort as
text, so it keeps a copy of the lines), and a job that fits unsorted fits sorted."""
import pytest
import torch

from unitigcoarsening_b200 import Compactor, synth
from unitigcoarsening_b200.api import UCError

pytestmark = pytest.mark.gpu

MIB = 1 << 20
EBUDGET = "HBM budget"


@pytest.mark.parametrize("k", [21, 31, 47, 63])
@pytest.mark.parametrize("warp_capacity", [0, 1])
def test_scratch_within_budget(comp, k, warp_capacity):
    n = 4_000_000
    spec = synth.GenomeSpec(length=n, gc=0.41, seed=k, snp_rate=0.001)
    text = synth.make_text(spec, k, "cuda")
    out = torch.empty(comp.output_bound(text.numel(), k), dtype=torch.uint8, device="cuda")

    def call(c, ordered):
        c.set_sorted_output(ordered)
        c.set_tuning(warp_capacity=warp_capacity)
        try:
            return c.compact(text, k, 8, out=out)
        finally:
            c.set_sorted_output(False)
            c.set_tuning(warp_capacity=0)

    call(comp, False)  # (loads the kernels)
    want = call(comp, True).clone()
    torch.cuda.synchronize()
    fitted = {False: [], True: []}
    for mib in range(96, 96 + 32 * 24, 24):
        for ordered in (False, True):
            with Compactor(0, hbm_budget=mib * MIB) as c:
                torch.cuda.synchronize()
                before = torch.cuda.mem_get_info()[0]
                try:
                    got = call(c, ordered)
                except UCError as e:
                    assert EBUDGET in str(e)
                    got = None
                torch.cuda.synchronize()
                used = before - torch.cuda.mem_get_info()[0]
                assert used <= (mib + 8) * MIB, (mib, ordered, used / MIB)
                if got is not None:
                    fitted[ordered].append(mib)
                    if ordered:
                        assert torch.equal(got, want)
    assert fitted[False] == fitted[True]
    assert 0 < len(fitted[False]) < 32
