"""uc_emit with 2^31 k-mers and more: ids and member counts take all 32 bits."""
import pytest
import torch

from unitigcoarsening_b200 import Compactor

pytestmark = pytest.mark.gpu


def test_emit_past_31_bits(comp):
    """2^30 lines of two k-mers and one of one, at k = 2: keys 'A' + ACGT[v % 4],
    so the lines alternate between AAC and AGT."""
    n, k = (1 << 31) + 1, 2
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 100 << 30:
        pytest.skip("needs 100 GB of device memory")
    keys = torch.empty((n, 1), dtype=torch.int64, device="cuda")
    head = torch.empty(n, dtype=torch.int32, device="cuda")
    rank = torch.empty(n, dtype=torch.int32, device="cuda")
    step = 1 << 28
    for a in range(0, n, step):
        v = torch.arange(a, min(n, a + step), dtype=torch.int64, device="cuda")
        keys[a: a + step, 0] = (v & 3) << 2
        rank[a: a + step] = (v & 1).to(torch.int32)
        v &= ~1
        head[a: a + step] = torch.where(v < 1 << 31, v, v - (1 << 32)).to(torch.int32)
    del v
    with Compactor(0) as c:
        out = c.write_unitigs(keys, keys, head, rank, k)
    assert out.numel() == (n // 2) * 4 + 3
    lines = out[: (n // 2) * 4].view(torch.int32)
    want = torch.frombuffer(bytearray(b"AAC\nAGT\n"), dtype=torch.int32).cuda()
    assert bool((lines[0::2] == want[0]).all()) and bool((lines[1::2] == want[1]).all())
    assert out[-3:].cpu().numpy().tobytes() == b"AA\n"
    del keys, head, rank, out, lines
    torch.cuda.empty_cache()
