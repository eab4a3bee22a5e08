"""Performance cases: what a user of the unitig compactor has it do, through
the Python binding, from the smallest served job to a genome-sized one.

A case names its entry point (``op``), the genome model its k-mers come from
(``model``), the genome length (``bases``; about as many distinct canonical
k-mers, the count the same for every seed), k and l:

op           entry point                              in a user's program
===========  =======================================  ==============================
compact      Compactor.compact, sorted output         text in HBM -> unitig lines in HBM
host         Compactor.compact_host, sorted output    pinned host text -> pinned host lines
load         Compactor.load_kmers                     text -> packed keys
edges        Compactor.assemble_pruned_graph          keys -> kept successor/predecessor
contract     Compactor.coarsen_de_bruijn_full_cycle   edges -> (head, rank), pointer jumping
hec          the same with CONTRACT_HEC               the reference's own matching
emit         Compactor.write_unitigs                  (head, rank) -> unitig lines

The whole-job cases run with sorted output, the mode whose bytes are the same
from run to run; without it (and in batches and the server) the lines come in
an order that changes from run to run, so two runs cannot be compared byte by
byte.  Both modes run the same pack, bucket, tile and stitch kernels.  The
phase entry points are deterministic as they are.

One context serves all jobs of a kind, as in a program that compacts one job
after another.
"""
import math

import torch

from unitigcoarsening_b200 import api, synth

# Declared ranges: bases per op, smallest and largest.  The lower end is the
# smallest served job (10k k-mers); the upper end of "compact" is a job of
# 8 GB of text (4 GB at two key words).
RANGES = {
    "compact": (10_000, 200_000_000),
    "host": (10_000, 16_000_000),
    "load": (10_000, 64_000_000),
    "edges": (10_000, 32_000_000),
    "contract": (10_000, 32_000_000),
    "hec": (10_000, 4_000_000),
    "emit": (10_000, 32_000_000),
}

# k with one key word and with two; 31 and 63 are the widths the reference is
# run with most, 15 mod 16 the ones it handles, the rest the common odd sizes
# of k-mer counters.
K_ONE = (31, 31, 21, 25, 27)
K_TWO = (63, 63, 47, 41, 55)


def listed():
    return [
        # the smallest request of the serving workload: latency and launches
        dict(name="compact_10k_k31", op="compact", model="served", bases=10_000, k=31, l=8),
        # the small plain job: a bacterial-sized genome with a few bubbles
        dict(name="compact_1M_k31", op="compact", model="small", bases=1_000_000, k=31, l=8),
        # a KMC dump as it comes (k-mer, tab, count): the general line layout
        dict(name="compact_5M_k21_counts", op="compact", model="counts", bases=5_234_567, k=21, l=8),
        # a mid-sized served job with two key words at an odd k
        dict(name="compact_12M_k47", op="compact", model="served", bases=12_345_679, k=47, l=9),
        # the wide-key job: tandem repeats, cycles and all
        dict(name="compact_64M_k63", op="compact", model="wide", bases=64_000_000, k=63, l=8),
        # the largest: a 256 Mbp genome with repeat families and SNPs
        dict(name="compact_256M_k31", op="compact", model="scale", bases=256_000_000, k=31, l=8),
        # one job host to host: PCIe both ways around the same path
        dict(name="host_3M_k31", op="host", model="batched", bases=3_000_000, k=31, l=8),
        # the phases one by one, as a program built on the reference's steps calls them
        dict(name="load_40M_k31", op="load", model="scale", bases=40_000_000, k=31, l=8),
        dict(name="edges_16M_k31", op="edges", model="scale", bases=16_000_000, k=31, l=8),
        dict(name="contract_16M_k31", op="contract", model="scale", bases=16_000_000, k=31, l=8),
        dict(name="hec_2M_k63", op="hec", model="wide", bases=2_000_003, k=63, l=8),
        dict(name="emit_16M_k31", op="emit", model="scale", bases=16_000_000, k=31, l=8),
    ]


def draw(rng):
    op = rng.choice(("compact", "compact", "compact", "compact", "host", "load", "edges", "contract", "hec",
                     "emit"))
    lo, hi = RANGES[op]
    two = rng.random() < 0.4
    if two:
        hi = min(hi, 50_000_000)
    bases = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    model = rng.choice(("served", "batched", "scale", "wide", "small"))
    if op in ("compact", "load") and bases < 40_000_000 and rng.random() < 0.2:
        model = "counts"
    return dict(op=op, model=model, bases=bases, k=rng.choice(K_TWO if two else K_ONE), l=rng.choice((8, 8, 9, 10)))


def genome(case, bases, seed):
    """The genome models of the library's generator, by name."""
    model = case["model"]
    if model == "small":    # uniform bases, SNP bubbles
        return synth.GenomeSpec(length=bases, gc=0.5, seed=seed, snp_count=max(1, bases // 5000))
    if model == "scale":    # 41% GC, repeat families, SNPs
        return synth.scale_plain(length=bases, seed=seed)
    if model == "wide":     # tandem repeats, SNPs
        return synth.wide_k(length=bases, seed=seed)
    if model == "batched":  # SNP-rich, GC away from a half
        return synth.GenomeSpec(length=bases, gc=0.3 + 0.4 * (seed % 97) / 96, seed=seed, snp_rate=0.002)
    # served, counts
    return synth.GenomeSpec(length=bases, gc=0.3 + 0.4 * (seed % 89) / 88, seed=seed, snp_rate=0.001)


def kmer_count(case):
    """k-mers of a case, the same for every seed: about what its genome model
    gives (each SNP adds k of them, repeats take some away)."""
    b, k = case["bases"], case["k"]
    snp = {"small": 0.0002, "scale": 0.001, "wide": 0.0005, "batched": 0.002}.get(case["model"], 0.001)
    lost = {"wide": 0.04, "scale": 0.01}.get(case["model"], 0.005)
    return int(b * (1 - lost + 0.95 * snp * k))


def kmers_of(case, seed):
    """The case's k-mers, shuffled: those of its genome, less the few past the
    count (a counter's cut-off) or with those of a small second sequence (a
    contamination) where the genome has fewer."""
    n, k = kmer_count(case), case["k"]
    kmers = synth.kmer_set(genome(case, case["bases"], seed), k, "cuda")
    extra = 1
    while kmers.shape[0] < n:
        spec = synth.GenomeSpec(length=2 * (n - kmers.shape[0]) + 1000, gc=0.45, seed=seed + 7_777_777 * extra)
        more = synth.kmer_set(spec, k, "cuda")[: n - kmers.shape[0]]
        both = torch.cat([kmers, more])
        both = torch.unique(both) if both.dim() == 1 else synth._unique_rows(both)
        kmers = synth.shuffle(both, seed)
        extra += 1
    return kmers[:n]


def dump_text(kmers, k):
    """The text of a k-mer counter's dump: k-mer, tab, count (1 to 99)."""
    n = kmers.shape[0]
    rows = torch.empty((n, k + 4), dtype=torch.uint8, device=kmers.device)
    rows[:, :k] = synth.kmers_to_lines(kmers, k)[:, :k]
    mix = kmers if kmers.dim() == 1 else kmers[:, 0] ^ kmers[:, 1]
    count = (mix ^ (mix >> 17)).remainder(99) + 1
    rows[:, k] = ord("\t")
    rows[:, k + 1] = (count // 10 + ord("0")).to(torch.uint8)
    rows[:, k + 2] = (count % 10 + ord("0")).to(torch.uint8)
    rows[:, k + 3] = ord("\n")
    keep = torch.ones_like(rows, dtype=torch.bool)
    keep[:, k + 1] = count >= 10
    header = torch.tensor(list(f"{n}\n".encode()), dtype=torch.uint8, device=kmers.device)
    return torch.cat([header, rows[keep]])


_contexts = {}


def context(sort_lines):
    """The program's context: one for whole jobs, one for the phases."""
    if sort_lines not in _contexts:
        c = api.Compactor(torch.cuda.current_device())
        c.set_sorted_output(sort_lines)
        _contexts[sort_lines] = c
    return _contexts[sort_lines]


def prepare(case, seed):
    op, k, l = case["op"], case["k"], case["l"]
    kmers = kmers_of(case, seed)
    n = kmers.shape[0]
    text = dump_text(kmers, k) if case["model"] == "counts" else synth.format_text(kmers, k)
    del kmers
    if text.numel() > 1 << 30:
        torch.cuda.empty_cache()  # the generator's temporaries: the library allocates its own memory
    whole = op in ("compact", "host")
    c = context(whole)
    s = dict(op=op, k=k, l=l, c=c)
    cap = c.output_bound(n * (k + 4) + 32, k)  # any line layout of these k-mers
    if op == "compact":
        s["text"] = text
        s["out"] = torch.zeros(cap, dtype=torch.uint8, device="cuda")
    elif op == "host":
        s["text"] = text.cpu().pin_memory()
        s["out"] = torch.zeros(cap, dtype=torch.uint8, pin_memory=True)
    elif op == "load":
        s["text"] = text
    else:
        s["keys"] = c.load_kmers(text, k)
        if op in ("contract", "hec", "emit"):
            s["succ"], s["pred"] = c.assemble_pruned_graph(s["keys"], k, l)
        if op == "emit":
            s["head"], s["rank"], _ = c.coarsen_de_bruijn_full_cycle(s["keys"], s["succ"], s["pred"], k)
            s["out"] = torch.zeros(n * (k + 1), dtype=torch.uint8, device="cuda")
    return s


def run(s):
    """One call.  Lines come in the program's own buffer, with their length."""
    op, c, k, l = s["op"], s["c"], s["k"], s["l"]
    if op == "compact":
        lines = c.compact(s["text"], k, l, out=s["out"])
        return {"lines": s["out"], "bytes": lines.numel()}
    if op == "host":
        lines = c.compact_host(s["text"], k, l, out=s["out"])
        return {"lines": s["out"], "bytes": lines.numel()}
    if op == "load":
        return c.load_kmers(s["text"], k)
    if op == "edges":
        return c.assemble_pruned_graph(s["keys"], k, l)
    if op in ("contract", "hec"):
        method = api.CONTRACT_HEC if op == "hec" else api.CONTRACT_POINTER_JUMP
        return c.coarsen_de_bruijn_full_cycle(s["keys"], s["succ"], s["pred"], k, method)
    # emit: the lines are collected in the program's buffer
    lines = c.write_unitigs(s["keys"], s["succ"], s["head"], s["rank"], k)
    s["out"][: lines.numel()] = lines
    return {"lines": s["out"], "bytes": lines.numel()}


def work(case):
    """Inputs once and outputs once.  5 in 12 canonical k-mers start a unitig
    (the runs of one strand), so the lines hold about n * (1 + 5 k / 12)
    bytes."""
    n, k = kmer_count(case), case["k"]
    key = 8 * api.key_words(k)
    text = n * (k + 1 + (3 if case["model"] == "counts" else 0))
    lines = n * (1 + 5 * k / 12)
    b = {
        "compact": text + lines,
        "host": text + lines,
        "load": text + n * key,
        "edges": n * key + 8 * n,
        "contract": 8 * n + 8 * n,   # succ, pred -> head, rank
        "hec": 8 * n + 8 * n,
        "emit": n * key + 8 * n + lines,
    }[case["op"]]
    return {"bytes": float(b), "flops": 0.0}


def exact(case, seed):
    """Every output is whole bytes or integers: nothing is rounded."""
    return None
