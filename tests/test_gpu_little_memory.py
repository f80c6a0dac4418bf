"""Calls on a device whose memory is nearly taken: what they need and cannot
have makes them fail cleanly or take another way to the same result, and what
they may take is bounded."""
import contextlib
import gc

import numpy as np
import pytest

import swapgb

pytestmark = pytest.mark.gpu

MB = 1 << 20


class _Rest:
    """What is left of the device's memory."""

    def __init__(self, steps):
        self.steps = steps

    def more(self):
        """One step more of it."""
        import torch
        self.steps.pop()
        torch.cuda.empty_cache()


@contextlib.contextmanager
def little_memory(left, step=0, steps=0):
    """Takes the device's free memory but `left` bytes, the last of it in
    `steps` blocks of `step` bytes that can be given back one by one."""
    import torch
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    blocks = []
    rest = _Rest([])
    try:
        take = torch.cuda.mem_get_info()[0] - left - step * steps
        blocks.append(torch.empty(take, dtype=torch.uint8, device="cuda"))
        for _ in range(steps):
            rest.steps.append(torch.empty(step, dtype=torch.uint8, device="cuda"))
        yield rest
    finally:
        blocks.clear()
        rest.steps.clear()
        torch.cuda.empty_cache()


@pytest.mark.parametrize("writer", ["write_kmer_graph", "write_node_lines"])
def test_failed_text_leaves_the_earlier_file(writer, tmp_path):
    """From no room for any scratch to room for all, in steps smaller than the
    text: a call that fails, at whichever allocation, leaves the file of the
    earlier call as it was."""
    rng = np.random.default_rng(1)
    read = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 3_000_000)].tobytes()
    g = swapgb.Graph().build_reads(swapgb.Opts(k=31, cutoff=1), swapgb.reads_from_fasta(b">r\n" + read + b"\n", 31))
    path = tmp_path / "text"
    write = getattr(g, writer)
    write(path)
    want = path.read_bytes()
    earlier = b"the earlier file\n"
    step = 48 * MB
    assert len(want) > 2 * step
    failed = 0
    with little_memory(32 * MB, step, 24) as rest:
        while True:
            path.write_bytes(earlier)
            try:
                write(path)
            except swapgb.SwgError:
                failed += 1
                assert path.read_bytes() == earlier
                rest.more()
                continue
            break
    assert failed >= 3 and path.read_bytes() == want


def _random_reads(n_reads, length, genome, seed):
    """Reads of one length at random places of a random genome, packed one over
    another: the words, and every read's offset and length, on the device."""
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    words = torch.randint(-2**31, 2**31, ((genome + 15) // 16,), generator=gen, device="cuda", dtype=torch.int32)
    off = torch.randint(0, genome - length + 1, (n_reads,), generator=gen, device="cuda")
    return words, off, torch.full((n_reads,), length, device="cuda", dtype=torch.int32)


def _build(g, opts, reads):
    import torch
    words, off, length = reads
    torch.cuda.synchronize()
    return g.build_device(opts, words.data_ptr(), words.numel(), off.data_ptr(), length.data_ptr(), off.numel())


@pytest.mark.parametrize("k,length,occurrences", [(31, 31, 25_000_000), (21, 22, 20_000_000), (31, 33, 25_000_000),
                                                  (21, 100, 24_000_000), (31, 31, 2_000_000), (31, 31, 70_000_000)])
def test_workspace_of_short_reads_is_bounded(k, length, occurrences):
    """53 bytes a k-mer occurrence and 64 MiB, the output included, however
    many super-k-mers a read's k-mers make."""
    import torch
    reads = _random_reads(occurrences // (length - k + 1), length, 1_000_000, k + length)
    g = swapgb.Graph()
    swapgb.Graph().build_reads(swapgb.Opts(k=21, cutoff=1), swapgb.reads_from_fasta(b">r\n" + b"ACGT" * 20 + b"\n", 21))
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    _build(g, swapgb.Opts(k=k, cutoff=2), reads)
    held = before - torch.cuda.mem_get_info()[0]
    # a read's place in the build's prefix and scan arrays (8 B), tables of the buckets, allocations rounded up to 2 MiB
    assert held <= 53 * occurrences + 64 * MB + 9 * reads[1].numel() + 64 * MB
    want = swapgb.Graph()
    _build(want, swapgb.Opts(k=k, cutoff=2, algorithm=swapgb.ALGO_DIRECT), reads)
    assert g.distinct() == want.distinct() > 500_000  # (reads of k bases have no arcs: no k-molecule stays)
    for a, b in zip(g.copy_out(), want.copy_out()):
        assert np.array_equal(a, b)


def test_sorted_fetch_keeps_to_the_budget():
    """The scratch of a fetch's sort (144 MB here) is charged to the server's
    budget, or the host sorts."""
    import torch
    rng = np.random.default_rng(2)
    read = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 1_000_000)].tobytes()
    reads = swapgb.reads_from_fasta(b">r\n" + read + b"\n", 31)
    want = swapgb.Graph().build_reads(swapgb.Opts(k=31, cutoff=1), reads).copy_out(sorted=True)
    for budget, most in ((100 * MB, 100 * MB // 16), (4 << 30, 256 * MB)):
        with_budget = swapgb.Server(memory_budget=budget, workers=1)
        ticket = with_budget.submit(reads, 31, 1)
        with_budget.wait(ticket, 60.0)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        keys, mult = with_budget.fetch(ticket)
        torch.cuda.synchronize()
        assert before - torch.cuda.mem_get_info()[0] <= most + 4 * MB
        assert with_budget.stats()["bytes_reserved"] == 0
        assert np.array_equal(keys, want[0]) and np.array_equal(mult, want[1])
        with_budget.close()


def _same(g, k, cutoff, reads):
    want = swapgb.Graph()
    _build(want, swapgb.Opts(k=k, cutoff=cutoff, algorithm=swapgb.ALGO_DIRECT), reads)
    assert g.size() == want.size() > 0
    for a, b in zip(g.copy_out(), want.copy_out()):
        assert np.array_equal(a, b)


# 12.7M occurrences in reads of 100 bases at k = 31: super-k-mer records take
# 409 MiB in regions of one size, 139 MiB in sampled ones, single occurrences
# 291 MiB (204 MB counted exactly); the first output 24 MiB.
N_READS = 181_429
BUCKETED = dict(k=31, algorithm=swapgb.ALGO_BUCKETED)


def test_regions_that_cannot_be_allocated():
    """Regions of one size do not fit, sampled ones do; then nothing fits, and
    the handle builds again once there is memory."""
    reads = _random_reads(N_READS, 100, 400_000, 1)
    g = swapgb.Graph()
    with little_memory(270 * MB):
        _build(g, swapgb.Opts(cutoff=2, **BUCKETED), reads)
    assert g.info()["estimate"] == 0
    _same(g, 31, 2, reads)
    g = swapgb.Graph()
    with little_memory(60 * MB):
        with pytest.raises(swapgb.SwgError) as e:
            _build(g, swapgb.Opts(cutoff=2, **BUCKETED), reads)
        assert e.value.status == 3
    _build(g, swapgb.Opts(cutoff=2, **BUCKETED), reads)
    _same(g, 31, 2, reads)


@pytest.mark.parametrize("genome,recounted", [(20_000, 0.0), (1_500_000, 1.0)])
def test_output_that_cannot_be_allocated(genome, recounted):
    """No room for the first guess of the output: the count alone says how much
    is needed, and that fits, or fits only once the records are given back and
    the build goes on over single occurrences."""
    reads = _random_reads(N_READS, 100, genome, 2)
    g = swapgb.Graph()
    _build(g, swapgb.Opts(cutoff=255, **BUCKETED), reads)
    with little_memory(8 * MB):
        _build(g, swapgb.Opts(cutoff=2, **BUCKETED), reads)
    assert g.info()["estimate"] == recounted
    _same(g, 31, 2, reads)
