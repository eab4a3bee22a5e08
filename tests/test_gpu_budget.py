"""Budgets that hold a job only with the shortest l-mers its buckets allow (fewer cross
k-mers, so smaller segment arrays): the job runs with those instead of being
refused.  Budgets just above what 4M k-mers of a uniform genome need that way;
with the l-mers taken otherwise they need 332, 385 and 398 MiB."""
import pytest
import torch

from unitigcoarsening_b200 import Compactor, api, synth

pytestmark = pytest.mark.gpu


def lines(t):
    return sorted(t.cpu().numpy().tobytes().split(b"\n"))


@pytest.mark.parametrize("k,mib,tuning,streamed", [
    (21, 312, dict(warp_capacity=1), False),
    (17, 340, dict(warp_capacity=1), False),
    (17, 374, {}, False),
    (17, 384, {}, True),
])
def test_budget_with_the_shortest_lmers(comp, k, mib, tuning, streamed):
    text = synth.make_text(synth.GenomeSpec(length=4_000_000, gc=0.5, seed=3, snp_rate=0.001), k, "cuda")
    want, st0 = comp.compact(text, k, 8, stats=True)
    with Compactor(0, hbm_budget=mib << 20) as c:
        c.set_tuning(**tuning)
        if streamed:
            c.set_streaming(api.STREAM_ALWAYS, 1 << 19, 1 << 18)
            got, st = c.compact_host(text.cpu(), k, 8, stats=True)
        else:
            got, st = c.compact(text, k, 8, stats=True)
            assert lines(comp.compact(text, k, 8)) == lines(want)
        assert st["l_used"] < st0["l_used"]
        assert lines(got) == lines(want)
        if not streamed:  # sorted output, and the same context again
            c.set_sorted_output(True)
            body = b"\n".join(x for x in lines(want) if x) + b"\n"
            assert c.compact(text, k, 8).cpu().numpy().tobytes() == body


def test_uploads_wait_for_the_retry(comp):
    """A sequence of host jobs whose uploads overlap: no text is replaced before
    the job that runs twice has read it twice."""
    k = 17
    texts = [synth.make_text(synth.GenomeSpec(length=4_000_000, gc=0.5, seed=s, snp_rate=0.001), k, "cuda").cpu().pin_memory()
             for s in (3, 4, 5)]
    want = [lines(comp.compact(x.cuda(), k, 8)) for x in texts]
    with Compactor(0, hbm_budget=374 << 20) as c:
        got = c.compact_host_many(texts, k, 8)
        assert [lines(torch.as_tensor(x)) for x in got] == want
