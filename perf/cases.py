"""Performance cases of the k-mer graph builder: what its users have it do.

A case is one pass through public entry points on seeded synthetic reads: a
uniform random genome (optionally with repeat families and tandem repeats),
reads from both strands with substitution errors, as every workload of this
repository has them. The kinds:

  host      packed reads in host memory -> graph on the host, sorted by key
            (Graph.build, Graph.copy_out): a program that builds one small
            graph and uses it on the CPU
  device    packed reads in device memory -> graph in device memory
            (Graph.build_device, Graph.device_view): the build alone
  fasta     FASTA text in pinned host memory -> graph in device memory
            (Graph.build_fasta): framing, packing and build in one call
  adjacency FASTA text -> graph -> kmerGraph.txt, what `swap -s` does
            (Graph.build_fasta, Graph.write_kmer_graph)
  batch     many samples of uneven size in one build, every sample's graph
            copied out (Graph.build_batch, Graph.batch_copy_out)
  serve     a burst of requests of uneven size, k and cutoff to the request
            server, every result fetched (Server)
  merge     the merge of semi-extended k-molecules of a built graph
            (Graph.merge, Graph.merged_text)
  contigs   reads in device memory -> graph -> merge -> tips, re-merge, low
            coverage, re-merge, what `swap -d` and the contig stage do

Graphs that stay on the device are unordered; the passes put them in key
order with a device sort, as a program that compares or joins graphs does.
"""
from __future__ import annotations

import math
import random
import sys
import tempfile
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "swap-assembler_gb300"))

import swapgb  # noqa: E402

HEADER = 10  # ">" + 8 digits + newline
CHUNK = 32 << 20  # padded bases generated at a time


def _case(name, kind, genome, coverage, read_min, read_max, sub, k, cutoff, repeats=False, samples=1):
    return dict(name=name, kind=kind, genome=genome, coverage=coverage, read_min=read_min, read_max=read_max,
                sub=sub, k=k, cutoff=cutoff, repeats=repeats, samples=samples)


def listed() -> list[dict]:
    return [
        # a plasmid or an amplicon, as the known-answer tests build them: latency and launches
        _case("host_plasmid", "host", 3_001, 20.0, 100, 100, 0.005, 21, 2),
        # a virus or phage, quality-trimmed reads of uneven length
        _case("host_trimmed_150k", "host", 150_001, 40.0, 36, 151, 0.005, 25, 3),
        # the plain sample: 1 Mbp at 30x, 300k reads of 100 bp
        _case("device_1m", "device", 1_000_000, 30.0, 100, 100, 0.005, 21, 2),
        # the same sample from its FASTA text to the adjacency file
        _case("adjacency_1m", "adjacency", 1_000_000, 30.0, 100, 100, 0.005, 21, 2),
        # the large single sample: 5 Mbp at 50x, 2.5M reads of 100 bp, 1% errors
        _case("device_5m", "device", 5_000_000, 50.0, 100, 100, 0.01, 31, 5),
        # the same sample from its FASTA text (long enough to be streamed in pieces)
        _case("fasta_5m", "fasta", 5_000_000, 50.0, 100, 100, 0.01, 31, 5),
        # the skewed sample: 100 Mbp with repeat families and tandem repeats, 20M reads of 150 bp
        _case("device_skewed_100m", "device", 100_000_000, 30.0, 150, 150, 0.005, 31, 3, repeats=True),
        # accurate long reads of a bacterium
        _case("device_long_reads", "device", 4_600_001, 40.0, 3_000, 15_000, 0.002, 31, 5),
        # a batch of samples as the batched workload draws them (k=27, c=3)
        _case("batch_24", "batch", 2_000_000, 60.0, 75, 250, 0.005, 27, 3, samples=24),
        # a burst of served requests, k and cutoff drawn per request
        _case("serve_24", "serve", 400_000, 60.0, 75, 250, 0.005, 31, 3, samples=24),
        # the merge of the large sample's graph: few long chains
        _case("merge_5m", "merge", 5_000_000, 50.0, 100, 100, 0.01, 31, 5),
        # the whole device pipeline on a graph with many branches left by errors
        _case("contigs_1m", "contigs", 1_000_000, 30.0, 100, 100, 0.005, 21, 2),
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng) -> dict:
    kind = rng.choice(["host", "device", "device", "fasta", "adjacency", "batch", "serve", "merge", "contigs"])
    genome = {"host": (1_500, 400_000), "device": (20_000, 50_000_000), "fasta": (5_000, 20_000_000),
              "adjacency": (5_000, 1_500_000), "batch": (50_000, 2_000_000), "serve": (50_000, 400_000),
              "merge": (20_000, 20_000_000), "contigs": (20_000, 3_000_000)}[kind]
    genome = _log(rng, *genome)
    coverage = rng.uniform(10, 60)
    k = rng.choice([21, 25, 27, 31, 19, 23, 29])
    cutoff = rng.choice([2, 3, 5])
    lo = rng.choice([75, 100, 150, 250])
    hi = lo
    samples = 1
    repeats = False
    if kind in ("host", "device", "fasta") and rng.random() < 0.4:  # trimmed reads
        lo, hi = 36, rng.choice([101, 151, 251])
    if kind == "device":
        repeats = rng.random() < 0.3
        if rng.random() < 0.25:  # long reads
            genome, lo, hi = min(genome, 10_000_000), rng.choice([800, 2_000]), rng.choice([5_001, 15_000])
            coverage, repeats = min(coverage, 40.0), False
    if kind == "batch":
        samples, k, cutoff, lo, hi = rng.randint(2, 28), 27, 3, 75, 250
    if kind == "serve":
        samples, lo, hi = rng.randint(4, 28), 75, 250
    if kind in ("merge", "contigs"):
        coverage = max(coverage, 20.0)
    return {f: v for f, v in _case("", kind, genome, round(coverage, 2), lo, hi, round(rng.uniform(0.001, 0.01), 5),
                                   k, cutoff, repeats, samples).items() if f != "name"}


# ---- inputs ---------------------------------------------------------------

def _rand(n, high, gen, dtype=torch.int64):
    return torch.randint(0, high, (n,), generator=gen, device="cuda", dtype=dtype)


def _genome(L, repeats, gen, rng):
    """Uniform bases (0..3); with repeats, 5% repeat families (units of 1-5
    kbp, log-uniform, 2-200 copies at 1% divergence) and 2% tandem repeats of
    2-6 bp units."""
    g = _rand(L, 4, gen, torch.uint8)
    if not repeats:
        return g
    placed, want = 0, L * 5 // 100
    while placed < want:
        unit = min(_log(rng, 1_000, 5_000), max(64, L // 20))
        copies = max(2, min(rng.randint(2, 200), (want - placed) // unit + 1))
        base = _rand(unit, 4, gen, torch.uint8).repeat(copies)
        mutated = torch.rand(base.numel(), generator=gen, device="cuda") < 0.01
        base = torch.where(mutated, _rand(base.numel(), 4, gen, torch.uint8), base)
        at = torch.tensor([rng.randrange(L // unit) for _ in range(copies)], device="cuda").unique()
        at = (at[:, None] * unit + torch.arange(unit, device="cuda")).reshape(-1)
        g[at] = base[:at.numel()]
        placed += unit * copies
    span = min(512, L)
    n = max(1, L * 2 // 100 // span)
    units = _rand(n * 6, 4, gen, torch.uint8).view(n, 6)
    period = _rand(n, 5, gen) + 2
    at = torch.randperm(L // span, generator=gen, device="cuda")[:n]
    pos = torch.arange(span, device="cuda")
    g[(at[:, None] * span + pos).reshape(-1)] = units[:at.numel()].gather(
        1, pos[None, :] % period[:at.numel(), None]).reshape(-1)
    return g


def _reads(c, gen, rng, fasta):
    """Reads of the case: as FASTA text (uint8 tensor), or packed as the
    library's framing packs them (16 bases a word, first base on top, every
    read from a word boundary): words, offsets, lengths. Device tensors."""
    g = _genome(c["genome"], c["repeats"], gen, rng)
    hi = min(c["read_max"], c["genome"])
    lo = min(c["read_min"], hi)
    n = max(1, int(c["coverage"] * c["genome"] / ((lo + hi) / 2)))
    lens = torch.full((n,), hi, device="cuda") if lo == hi else _rand(n, hi - lo + 1, gen) + lo
    begin = (torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) * (c["genome"] - lens + 1)).long()
    flip = _rand(n, 2, gen, torch.uint8)
    room = HEADER + lens + 1 if fasta else (lens + 15) // 16 * 16
    off = torch.cumsum(room, 0) - room
    total = int(off[-1] + room[-1])
    out = torch.empty(total if fasta else total // 16, device="cuda", dtype=torch.uint8 if fasta else torch.int32)
    letters = torch.tensor(list(b"ACGT"), device="cuda", dtype=torch.uint8)
    r0 = 0
    step = max(1, CHUNK // int(room.max()))
    while r0 < n:
        r1 = min(n, r0 + step)
        o0, o1 = int(off[r0]), int(off[r1 - 1] + room[r1 - 1])
        rid = torch.repeat_interleave(torch.arange(r0, r1, device="cuda"), room[r0:r1], output_size=o1 - o0)
        pos = torch.arange(o0, o1, device="cuda") - off[rid]
        if fasta:
            head = pos < HEADER
            pos = pos - HEADER
        inside = (pos >= 0) & (pos < lens[rid])
        rev = flip[rid].bool()
        at = begin[rid] + torch.where(rev, lens[rid] - 1 - pos, pos)
        b = g[at.clamp_(0, c["genome"] - 1)]
        b = torch.where(rev, 3 - b, b)
        err = torch.rand(o1 - o0, generator=gen, device="cuda") < c["sub"]
        b = torch.where(err, (b + 1 + _rand(o1 - o0, 3, gen, torch.uint8)) & 3, b)
        if fasta:
            div = 10 ** (8 - (pos + HEADER).clamp(1, 8))
            digit = (48 + rid // div % 10).to(torch.uint8)
            text = torch.where(inside, letters[b.long()], 10)
            text = torch.where(head, digit, text)
            text = torch.where(pos == -HEADER, 62, text)
            out[o0:o1] = torch.where(pos == -1, 10, text)
        else:
            b = torch.where(inside, b, 0).view(-1, 16).to(torch.int64)
            sh = torch.arange(30, -1, -2, device="cuda")
            out[o0 // 16:o1 // 16] = (b << sh).sum(1).to(torch.int32)
        r0 = r1
    if fasta:
        return out
    return out, off, lens.to(torch.int32)


def _capacity(c):
    """K-molecules that the arrays a program keeps for the case's graph hold:
    the genome's and, at the lowest cutoff, those of errors seen twice."""
    return (4 if c["cutoff"] <= 2 else 2) * c["genome"] + 4096


def _samples(c, gen):
    """Host reads of a batch's or a burst's samples (genome log-uniform up to
    the case's, coverage 10x up to the case's, read length one of four; the
    same sizes for every seed), and each one's k, cutoff and capacity."""
    out = []
    rng = random.Random(c["samples"] * 1_000_003 + c["genome"])
    for _ in range(c["samples"]):
        length = rng.choice([v for v in (75, 100, 150, 250) if c["read_min"] <= v <= c["read_max"]])
        one = dict(c, genome=_log(rng, min(20_000, c["genome"]), c["genome"]),
                   coverage=rng.uniform(min(10.0, c["coverage"]), c["coverage"]), read_min=length, read_max=length)
        k = rng.choice([21, 25, 27, 31]) if c["kind"] == "serve" else c["k"]
        cut = rng.choice([2, 3, 5]) if c["kind"] == "serve" else c["cutoff"]
        text = _reads(one, gen, rng, True).cpu().numpy().tobytes()
        out.append(((swapgb.reads_from_fasta(text, k), k, cut), _capacity(dict(one, cutoff=cut))))
    return out


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    rng = random.Random(seed)
    c, kind = case, case["kind"]
    st = {"case": c, "stream": torch.cuda.Stream()}
    if kind in ("batch", "serve"):
        both = _samples(c, gen)
        st["samples"] = [one for one, _ in both]
        st["out"] = [(np.zeros(cap, np.uint64), np.zeros((cap, 8), np.uint8)) for _, cap in both]
    elif kind in ("fasta", "adjacency"):
        t = _reads(c, gen, rng, True)
        st["text"] = torch.empty(t.numel(), dtype=torch.uint8, pin_memory=True)
        st["text"].copy_(t)
    else:
        st["reads"] = _reads(c, gen, rng, False)
        if kind == "host":
            p, o, n = (t.cpu().numpy() for t in st.pop("reads"))
            st["host"] = p.view(np.uint32), o.view(np.uint64), n.view(np.uint32)
            st["out"] = [(np.zeros(_capacity(c), np.uint64), np.zeros((_capacity(c), 8), np.uint8))]
    if kind in ("device", "fasta"):
        st["out"] = torch.zeros(2, _capacity(c), dtype=torch.int64, device="cuda")
    if kind in ("adjacency", "merge", "contigs"):
        st["out"] = np.zeros((_capacity(c) * 90 if kind == "adjacency" else 24 * c["genome"]) + (1 << 16), np.uint8)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()  # the library allocates its own device memory
    if kind == "serve":
        st["server"] = swapgb.Server()
    else:
        st["graph"] = swapgb.Graph()
        st["opts"] = swapgb.Opts(k=c["k"], cutoff=c["cutoff"], stream=st["stream"].cuda_stream)
    if kind == "adjacency":
        st["dir"] = tempfile.TemporaryDirectory()
    if kind == "merge":
        _build_device(st)
        del st["reads"]
    return st


# ---- passes ---------------------------------------------------------------

class _DeviceArray:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<i8", data=(ptr, False), version=3)


def _build_device(st):
    p, o, n = st["reads"]
    st["graph"].build_device(st["opts"], p.data_ptr(), p.numel(), o.data_ptr(), n.data_ptr(), o.numel())


def _device_graph(st):
    """The graph in key order, in the program's own device arrays (keys; the 8
    multiplicities of each), and its size."""
    k, m, n = st["graph"].device_view()
    if n:
        with torch.cuda.stream(st["stream"]):
            fit = min(n, st["out"].shape[1])
            keys, order = torch.sort(torch.as_tensor(_DeviceArray(k, n), device="cuda"))
            st["out"][0, :fit] = keys[:fit]
            torch.index_select(torch.as_tensor(_DeviceArray(m, n), device="cuda"), 0, order[:fit],
                               out=st["out"][1, :fit])
    return st["out"], n


def _host_graph(out, graph):
    """A graph copied out by the library, in the program's own host arrays."""
    for kept, got in zip(out, graph):
        fit = min(len(kept), len(got))
        kept[:fit] = got[:fit]
    return out[0], out[1], len(graph[0])


def _host_bytes(out, data):
    fit = min(len(out), len(data))
    out[:fit] = data[:fit]
    return out, len(data)


def _merged(st):
    return _host_bytes(st["out"], np.frombuffer(st["graph"].merged_text(), dtype=np.uint8))


def run(state):
    st, kind = state, state["case"]["kind"]
    if kind == "serve":
        tickets = [st["server"].submit(*s) for s in st["samples"]]
        sizes = []
        for t, out in zip(tickets, st["out"]):
            st["server"].wait(t)
            sizes.append(_host_graph(out, st["server"].fetch(t))[2])
        return st["out"], np.array(sizes)
    g = st["graph"]
    if kind == "host":
        g.build(st["opts"], *st["host"])
        return _host_graph(st["out"][0], g.copy_out())
    if kind == "batch":
        g.build_batch(st["opts"], st["samples"])
        sizes = [_host_graph(out, g.batch_copy_out(i))[2] for i, out in enumerate(st["out"])]
        return st["out"], np.array(sizes)
    if kind == "merge":
        g.merge()
        return _merged(st)
    if kind in ("fasta", "adjacency"):
        g.build_fasta(st["opts"], (st["text"].data_ptr(), st["text"].numel()))
        if kind == "fasta":
            return _device_graph(st)
        path = Path(st["dir"].name) / "kmerGraph.txt"
        g.write_kmer_graph(str(path))
        return _host_bytes(st["out"], np.fromfile(path, dtype=np.uint8))
    _build_device(st)
    if kind == "device":
        return _device_graph(st)
    g.merge()
    counts = [g.remove_tips(), g.simplify(), g.remove_low_coverage(), g.simplify()]
    return _merged(st), np.array(counts)


def work(case):
    """Bytes: the reads (or the text, or the graph) once, the result once. A
    graph holds about one k-molecule (16 bytes) per base of the genome."""
    c = case
    n = c["coverage"] * c["genome"] / ((c["read_min"] + c["read_max"]) / 2)
    bases = c["coverage"] * c["genome"]
    graph = 16.0 * c["genome"]
    packed = bases / 4 + 12 * n
    text = bases + (HEADER + 1) * n
    kind = c["kind"]
    if kind in ("batch", "serve"):
        lo = min(20_000, c["genome"])
        mean = c["genome"] if lo == c["genome"] else (c["genome"] - lo) / math.log(c["genome"] / lo)
        cov = (min(10.0, c["coverage"]) + c["coverage"]) / 2
        return {"bytes": c["samples"] * mean * (cov / 4 + 12 * cov / 144 + 16), "flops": 0}
    if kind in ("host", "device"):
        return {"bytes": packed + graph, "flops": 0}
    if kind == "fasta":
        return {"bytes": text + graph, "flops": 0}
    if kind == "adjacency":  # about 130 characters a k-molecule at k = 31
        return {"bytes": text + c["genome"] * 4.2 * c["k"], "flops": 0}
    if kind == "merge":  # the graph; two strands of arc strings
        return {"bytes": graph + 2.0 * c["genome"], "flops": 0}
    return {"bytes": packed + 2.0 * c["genome"], "flops": 0}
