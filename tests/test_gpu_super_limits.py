"""Bucketed builds at the limits of their workspace: regions that are too
small, memory that is too little, records that are too many. The graph stays
exactly the one of the CPU restatement or of a build without the limit
(integers: the tolerance is zero)."""
import threading

import numpy as np
import pytest

import oracle
import swapgb
from test_gpu_super import _fasta, _random, _sampled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [0, 1])
def test_regions_outgrown_in_several_threads(shape):
    """Reads of one base outgrow their regions, and the build counts again: the
    counting kernels' blocks set the status that others of the launch read as
    they start. Several builds at once make blocks start late."""
    rng = np.random.default_rng(3 + shape)
    k = 21
    jobs = []
    for genome, n, alike in ((30_000, 10_000, 2_000), (200_000, 30_000, 9_000)):
        reads = [b"A" * 100] * alike + _sampled(rng, _random(rng, genome), n, [100])
        text = _fasta([reads[i] for i in rng.permutation(len(reads))])
        jobs.append((swapgb.reads_from_fasta(text, k), oracle.records(text, k, 2)))
    failed = []

    def work(reads, want):
        g = swapgb.Graph()
        for _ in range(25):
            try:
                g.build_reads(swapgb.Opts(k=k, cutoff=2, algorithm=swapgb.ALGO_BUCKETED, scatter_shape=shape), reads)
                if shape and g.info()["estimate"] != 1.0:
                    failed.append("nothing was outgrown")
                got = g.copy_out(sorted=True)
                if not (np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])):
                    failed.append("differs")
            except swapgb.SwgError as e:
                failed.append(str(e))

    threads = [threading.Thread(target=work, args=j) for j in jobs for _ in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed[:3]


@pytest.mark.parametrize("copies", [8_191, 8_192, 8_193, 9_216, 9_217])
def test_hot_bucket_from_8193_records(copies):
    """A bucket of more than 8192 records goes to the global-memory table, in
    chunks of 1024 records. Copies of one read: nothing else is in its buckets."""
    k = 21
    read = _random(np.random.default_rng(copies), k + 2)
    text = _fasta([read] * copies)
    g = swapgb.Graph().build_reads(swapgb.Opts(k=k, cutoff=2), swapgb.reads_from_fasta(text, k))
    assert (g.info()["waves"] >= 1) == (copies > 8_192)
    keys, mult = g.copy_out(sorted=True)
    okeys, omult = oracle.records(text, k, 2)
    assert keys.size == 3 and np.array_equal(keys, okeys) and np.array_equal(mult, omult)


def _view(ptr, n, shape=None):
    import torch

    class Array:
        __cuda_array_interface__ = dict(shape=(n,), typestr="<i8", data=(ptr, False), version=3)

    return torch.as_tensor(Array(), device="cuda")


def _sorted_graph(g):
    import torch
    k, m, n = g.device_view()
    keys, order = torch.sort(_view(k, n))
    return keys, _view(m, n)[order]


@pytest.mark.parametrize("k", [19, 21, 23, 25])
@pytest.mark.parametrize("occurrences", [280_000_000, 2_200_000_000])
def test_minimizers_of_large_builds(k, occurrences):
    """More than 256M occurrences, and more than 2G, take longer m-mers, in
    kernels of their own: the graph is the one of the build over single
    occurrences. Reads of k - 1 to k + 18 bases and more, from both strands of a
    random genome with some low-complexity stretches."""
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(k)
    genome = 16_000_000
    bases = torch.randint(0, 4, (genome,), generator=gen, device="cuda", dtype=torch.uint8)
    for i in range(8):
        at, unit = 1_000_000 * (2 * i + 1), torch.arange(i % 4 + 1, device="cuda", dtype=torch.uint8)
        bases[at:at + 600] = unit.repeat(600)[:600]
    bases = torch.cat([bases, 3 - bases.flip(0)])
    words = (bases.view(-1, 16).to(torch.int64) << torch.arange(30, -1, -2, device="cuda")).sum(1).to(torch.int32)
    lengths = torch.tensor([k - 1, k, k + 1, k + 16, k + 17, k + 18, 100, 133, 150, 151, 250, 400], device="cuda")
    n = int(occurrences / (lengths - k + 1).clamp(min=0).float().mean())
    length = lengths[torch.randint(0, lengths.numel(), (n,), generator=gen, device="cuda")]
    off = (torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) * (2 * genome - length)).long()
    length = length.to(torch.int32)
    torch.cuda.synchronize()
    got = []
    for shape in (0, 1):
        g = swapgb.Graph().build_device(swapgb.Opts(k=k, cutoff=2, algorithm=swapgb.ALGO_BUCKETED, scatter_shape=shape),
                                        words.data_ptr(), words.numel(), off.data_ptr(), length.data_ptr(), n)
        assert g.info()["occurrences"] > (2 << 30 if occurrences > 1 << 30 else 256 << 20)
        assert g.size() > 10_000_000
        got.append((g.distinct(), *_sorted_graph(g)))
        torch.cuda.synchronize()
    assert got[0][0] == got[1][0]
    assert torch.equal(got[0][1], got[1][1]) and torch.equal(got[0][2], got[1][2])


def _rows(rng, n, length):
    """FASTA text of n random reads of one length."""
    rows = np.empty((n, length + 3), np.uint8)
    rows[:, 0], rows[:, 1], rows[:, -1] = ord(">"), ord("\n"), ord("\n")
    rows[:, 2:-1] = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, (n, length), np.uint8)]
    return rows


@pytest.mark.parametrize("length,last", [(31, 0), (33, 0), (600, 0), (16_383, 0), (100, 16_384), (100, 40_000)])
def test_streamed_lengths(length, last):
    """Texts long enough to be streamed: reads whose super-k-mer records would
    take more memory than their occurrences, long reads, and one that is too
    long for a streamed piece's scan only at the end."""
    from test_gpu_stream import STREAM_MIN, assert_same
    rng = np.random.default_rng(length + last)
    rows = _rows(rng, (STREAM_MIN // 2) // (length + 3) + 1, length)
    text = rows.tobytes() * 2  # every read twice
    if last:
        text += (b">x\n" + _random(rng, last) + b"\n") * 2
    info = assert_same(text + b">y\n" + b"A" * 100 + b"\n", swapgb.Opts(k=31, cutoff=2, algorithm=swapgb.ALGO_BUCKETED))
    assert info["survivors"] > 0 or length == 31


def _order_for_one_bucket(keys, at):
    """A permutation that puts the smallest keys at the places `at`."""
    order = np.argsort(keys)
    rest = np.setdiff1d(np.arange(keys.size), at)
    perm = np.empty(keys.size, np.int64)
    perm[at] = order[:at.size]
    perm[rest] = np.random.default_rng(1).permutation(order[at.size:])
    return perm


def _reorder(g, perm):
    import torch
    k, m, n = g.device_view()
    p = torch.from_numpy(perm).cuda()
    for ptr in (k, m):
        v = _view(ptr, n)
        v.copy_(v[p])
    torch.cuda.synchronize()


@pytest.mark.parametrize("n", [8_192, 16_384, 100_000, 1 << 20])
def test_sorted_copy_with_a_full_bucket(n):
    """The sampled places (four a bucket of 512 records, at even strides) hold
    the smallest keys, so that nearly all records fall into the last bucket:
    more than its region takes, and the radix passes follow."""
    rng = np.random.default_rng(n)
    read = _random(rng, n + 30)
    g = swapgb.Graph().build_reads(swapgb.Opts(k=31, cutoff=1), swapgb.reads_from_fasta(b">r\n" + read + b"\n", 31))
    keys, mult = g.copy_out(sorted=False)
    assert keys.size == n
    count = 4 * ((n + 511) // 512)
    at = (np.arange(count, dtype=np.int64) * ((n << 20) // count)) >> 20
    _reorder(g, _order_for_one_bucket(keys, at))
    skeys, smult = g.copy_out(sorted=True)
    order = np.argsort(keys)
    assert np.array_equal(skeys, keys[order]) and np.array_equal(smult, mult[order])


@pytest.mark.parametrize("fragments", [4_096, 65_536])
def test_merge_lines_with_a_full_bucket(fragments):
    """The same for the merge's line sort. All nodes are lines here (fragments
    of k + 1 bases), listed by warps of 32 in any order, and the sampled places
    are multiples of 128: a warp's first lane has one of the smallest keys."""
    rng = np.random.default_rng(fragments)
    k = 31
    reads = [_random(rng, k + 1) for _ in range(fragments)]
    g = swapgb.Graph().build_reads(swapgb.Opts(k=k, cutoff=1), swapgb.reads_from_fasta(_fasta(reads), k))
    keys, mult = g.copy_out(sorted=False)
    assert keys.size == 2 * fragments
    want = oracle.merge_text(*oracle.records(_fasta(reads), k, 1), k)
    g.merge()
    assert g.merged_text() == want
    _reorder(g, _order_for_one_bucket(keys, np.arange(0, keys.size, 32)))
    g.merge()
    assert g.merge_info()["nodes"] == keys.size and g.merged_text() == want
