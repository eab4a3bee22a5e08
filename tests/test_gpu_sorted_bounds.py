"""Sorted output writes its lines and not one byte more, at every alignment of
the buffer, for lines that reach the sort as records, as text, and as long ones."""
import pytest
import torch

from tests.cases import random_seq, shuffled, sorted_lines, text_of, walk_kmers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [21, 31, 33, 63])
@pytest.mark.parametrize("warp_capacity", [0, 1])
@pytest.mark.parametrize("lengths", ["one", "tails", "long", "huge"])
def test_nothing_past_the_lines(comp, oracle, k, warp_capacity, lengths):
    lens = {"one": [k], "tails": [k + t for t in range(36)] * 30, "long": [k, k + 28, k + 29, 300, 16_384, 16_500] * 3,
            "huge": [k, 65_535, 65_536, 150_000, k + 5]}[lengths]
    kmers = []
    for i, m in enumerate(lens):
        kmers += walk_kmers(random_seq(m, 3000 * k + i), k)
    text = text_of(shuffled(kmers, 2))
    expect = b"".join(x + b"\n" for x in sorted_lines(oracle.compact(text, k)[0]))
    d = torch.frombuffer(bytearray(text), dtype=torch.uint8).cuda()
    buf = torch.empty(comp.output_bound(len(text), k) + 32, dtype=torch.uint8, device="cuda")
    comp.set_sorted_output(True)
    comp.set_tuning(warp_capacity=warp_capacity)
    try:
        for shift in range(17) if lengths != "huge" else (0, 3, 13):
            buf.fill_(0x55)
            m = comp.compact(d, k, 8, out=buf[shift:]).numel()
            assert buf[shift: shift + m].cpu().numpy().tobytes() == expect
            assert bool((buf[:shift] == 0x55).all()) and bool((buf[shift + m:] == 0x55).all())
    finally:
        comp.set_tuning(warp_capacity=0)
        comp.set_sorted_output(False)
