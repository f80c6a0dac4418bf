"""The bucketed build over super-k-mer records (runs of k-mers with one
minimizer): the graph equals the CPU restatement's, every multiplicity
included (integers: the tolerance is zero), at the edges of what the build
takes: every k it is built for, reads of k, k + 1 and k + 17 bases, lengths
around the cut into pieces (512) and past what a record's position holds
(16,383), any base offset, low-complexity and identical reads."""
import numpy as np
import pytest

import oracle
import swapgb

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _random(rng, n):
    return ACGT[rng.integers(0, 4, n)].tobytes()


def _fasta(reads):
    return b"".join(b">%d\n%s\n" % (i, r) for i, r in enumerate(reads))


def _sampled(rng, genome, n, lengths, err=0.004):
    """Reads of a genome, half of them from the other strand."""
    comp = bytes.maketrans(b"ACGT", b"TGCA")
    out = []
    for i in range(n):
        L = min(lengths[i % len(lengths)], len(genome))
        at = int(rng.integers(0, len(genome) - L + 1))
        r = np.frombuffer(genome[at:at + L], np.uint8).copy()
        bad = rng.random(L) < err
        r[bad] = ACGT[rng.integers(0, 4, int(bad.sum()))]
        r = r.tobytes()
        out.append(r if i & 1 else r.translate(comp)[::-1])
    return out


def _check(reads, k, c, **opts):
    text = _fasta(reads)
    g = swapgb.Graph().build_reads(swapgb.Opts(k=k, cutoff=c, **opts), swapgb.reads_from_fasta(text, k))
    assert g.info()["algorithm"] == swapgb.ALGO_BUCKETED
    assert g.info()["occurrences"] >= 600_000  # several buckets a block
    keys, mult = g.copy_out(sorted=True)
    okeys, omult = oracle.records(text, k, c)
    assert np.array_equal(keys, okeys) and np.array_equal(mult, omult)
    return g


@pytest.mark.parametrize("k", [19, 21, 23, 25, 27, 29, 31])
@pytest.mark.parametrize("c", [0, 1, 3, 255, 256])
def test_every_k_and_cutoff(k, c):
    rng = np.random.default_rng(100 * k + c)
    lengths = [k - 1, k, k + 1, k + 16, k + 17, k + 18, 100, 151, 250]
    _check(_sampled(rng, _random(rng, 40_000), 12_000, lengths), k, c)


@pytest.mark.parametrize("lengths", [[511, 512, 513], [2_000, 767, 31], [60, 16_384 + 31, 9_000]])
def test_long_reads(lengths):
    rng = np.random.default_rng(len(lengths) + lengths[0])
    n = 2_400_000 // (sum(lengths) // 3)
    _check(_sampled(rng, _random(rng, 60_000), n, lengths), 31, 2, algorithm=swapgb.ALGO_BUCKETED)


@pytest.mark.parametrize("k", [21, 31])
def test_low_complexity_and_identical_reads(k):
    """Runs longer than a record, records all equal (weights, clamped
    counters), buckets past the shared tables, saturated multiplicities."""
    rng = np.random.default_rng(k)
    one = _random(rng, 120)
    reads = _sampled(rng, _random(rng, 30_000), 4_000, [100])
    reads += [one] * 6_000 + [b"A" * 90] * 3_000 + [b"AC" * 60] * 3_000 + [b"ACGTTGCA" * 15] * 500
    reads += [b"ACG" * 40 + _random(rng, 30) for _ in range(2_000)]
    g = _check(reads, k, 2)
    assert (g.copy_out()[1] == 255).any()


@pytest.mark.parametrize("copies", [16_385, 17_408, 17_409, 60_000])
def test_hot_buckets(copies):
    """Buckets for the global-memory table, around a whole number of its chunks
    of 1024 records: copies of one short read, of another with one of three
    last bases, and of a read within a tandem repeat (equal k-molecules in one
    record, weights past 255)."""
    rng = np.random.default_rng(copies)
    k = 21
    hot = _random(rng, k + 2)
    other = _random(rng, k + 1)
    reads = [hot] * copies + [other[:k] + b"ACG"[i % 3:i % 3 + 1] for i in range(copies)] + [b"AC" * 30] * (copies // 10)
    reads += _sampled(rng, _random(rng, 40_000), 8_000, [100])
    reads = [reads[i] for i in rng.permutation(len(reads))]
    assert _check(reads, k, 2).info()["waves"] >= 1


@pytest.mark.parametrize("repeats", [0, 4_000])
@pytest.mark.parametrize("total", [1 << 20, 1024 * 3072, 1024 * 3072 + 1])
def test_regions_of_one_size(total, repeats):
    """Up to 1024 buckets (of 3072 occurrences on average) there is no second
    level; regions are of one size, unsampled, there and in somewhat larger
    builds; reads of one base repeated outgrow theirs and the build goes on with
    sampled ones."""
    rng = np.random.default_rng(9)
    k = 21
    reads = [b"A" * 100] * repeats
    left = total - 80 * repeats
    reads += _sampled(rng, _random(rng, 30_000), left // 80, [100])
    if left % 80:
        reads += [_random(rng, k - 1 + left % 80)]
    reads = [reads[i] for i in rng.permutation(len(reads))]
    g = _check(reads, k, 2)
    assert g.info()["occurrences"] == total


def test_few_survivors_and_many():
    """More survivors than the first output size (one per 8 occurrences):
    the count runs again into a larger one."""
    rng = np.random.default_rng(5)
    _check(_sampled(rng, _random(rng, 900_000), 15_000, [100], err=0.0), 25, 1)
    _check(_sampled(rng, _random(rng, 900_000), 15_000, [100], err=0.0), 25, 3)


@pytest.mark.parametrize("k", [23, 31])
def test_any_base_offset(k):
    """Reads packed one after another (any alignment in a word), in reverse
    order, overlapping, with the last one ending in the last word."""
    import torch
    rng = np.random.default_rng(7 + k)
    genome = _random(rng, 20_000)
    reads = _sampled(rng, genome, 9_000, [k, 77, 100, 133])
    codes = (np.frombuffer(b"".join(reads), np.uint8) >> 1) ^ (np.frombuffer(b"".join(reads), np.uint8) >> 2)
    codes = (codes & 3).astype(np.uint32)
    lens = np.array([len(r) for r in reads], np.uint32)
    off = (np.cumsum(lens.astype(np.uint64)) - lens).astype(np.uint64)
    pad = np.zeros(-len(codes) % 16, np.uint32)
    words = (np.concatenate([codes, pad]).reshape(-1, 16) << np.arange(30, -1, -2, dtype=np.uint32)).sum(1, dtype=np.uint32)
    off = np.concatenate([off[::-1], off[:500]])  # some reads twice
    lens = np.concatenate([lens[::-1], lens[:500]])
    text = _fasta(reads[::-1] + reads[:500])
    p, o, ln = (torch.from_numpy(x.view(t).copy()).cuda() for x, t in
                ((words, np.int32), (off, np.int64), (lens, np.int32)))
    torch.cuda.synchronize()
    g = swapgb.Graph().build_device(swapgb.Opts(k=k, cutoff=2), p.data_ptr(), p.numel(), o.data_ptr(), ln.data_ptr(),
                                    o.numel())
    assert g.info()["algorithm"] == swapgb.ALGO_BUCKETED and g.info()["occurrences"] >= 500_000
    keys, mult = g.copy_out(sorted=True)
    okeys, omult = oracle.records(text, k, 2)
    assert np.array_equal(keys, okeys) and np.array_equal(mult, omult)


@pytest.mark.parametrize("k,lengths", [(21, [100, 150]), (27, [75, 700])])
def test_batch_of_one_k(k, lengths):
    """Samples of one k share a build over tagged records (long reads in
    pieces); each sample equals the restatement on it alone."""
    rng = np.random.default_rng(k)
    texts = [_fasta(_sampled(rng, _random(rng, 3_000 + 500 * i), 1_500 + 100 * i, lengths)) for i in range(9)]
    texts.append(_fasta([b"A" * 100] * 1_500))
    batch = [(swapgb.reads_from_fasta(t, k), k, i % 4) for i, t in enumerate(texts)]
    g = swapgb.Graph().build_batch(swapgb.Opts(), batch)
    assert g.info()["algorithm"] == swapgb.ALGO_BUCKETED and g.info()["occurrences"] >= 600_000
    for i, t in enumerate(texts):
        keys, mult = g.batch_copy_out(i)
        okeys, omult = oracle.records(t, k, i % 4)
        assert np.array_equal(keys, okeys) and np.array_equal(mult, omult), i


def test_builds_of_several_threads():
    """Builds of different sizes (and so kernels with different shared memory)
    from several threads, each with its own handle: every one succeeds."""
    import threading
    rng = np.random.default_rng(11)
    jobs = []
    for genome, n, k in [(5_000, 8_000, 31), (400_000, 150_000, 31), (60_000, 30_000, 21), (400_000, 150_000, 21)]:
        text = _fasta(_sampled(rng, _random(rng, genome), n, [100]))
        reads = swapgb.reads_from_fasta(text, k)
        jobs.append((k, reads, swapgb.Graph().build_reads(swapgb.Opts(k=k, cutoff=2), reads).copy_out()))
    failed = []

    def work(k, reads, want):
        g = swapgb.Graph()
        for _ in range(40):
            try:
                got = g.build_reads(swapgb.Opts(k=k, cutoff=2), reads).copy_out()
                if not (np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])):
                    failed.append("differs")
            except swapgb.SwgError as e:
                failed.append(str(e))

    threads = [threading.Thread(target=work, args=j) for j in jobs for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed[:3]
