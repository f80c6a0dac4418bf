"""Sorted copies of a graph to the host (ordered on the device) are the
unsorted copy in key order, exactly: one block's sort and its limit (4096
records), the radix passes' tile edges, every number of passes (k)."""
import numpy as np
import pytest

import swapgb

pytestmark = pytest.mark.gpu


def _check(g, n=None):
    keys, mult = g.copy_out(sorted=False)
    skeys, smult = g.copy_out(sorted=True)
    if n is not None:
        assert keys.size == n
    order = np.argsort(keys)
    assert np.array_equal(skeys, keys[order]) and np.array_equal(smult, mult[order])
    again = g.copy_out(sorted=False)
    assert np.array_equal(again[0], keys) and np.array_equal(again[1], mult)  # the graph's own order stays


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1000, 1022, 1023, 1024, 1025, 2047, 2048, 2049, 4095, 4096, 4097, 8191, 8192, 8193, 70_001, 1_048_575, 1_048_576,
                               1_048_577, 1_503_001])
def test_sizes(n):
    rng = np.random.default_rng(n)
    read = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, n + 31)].tobytes()
    reads = swapgb.reads_from_fasta(b">r\n" + read + b"\n", 31)  # n + 1 distinct k-molecules
    for algo in (swapgb.ALGO_BUCKETED, swapgb.ALGO_DIRECT) if n < 10_000 else (swapgb.ALGO_DIRECT,):
        _check(swapgb.Graph().build_reads(swapgb.Opts(k=31, cutoff=1, algorithm=algo), reads), n + 1)


@pytest.mark.parametrize("k", [1, 3, 4, 5, 8, 9, 12, 13, 16, 17, 20, 21, 24, 25, 28, 29, 31])
def test_every_number_of_passes(k):
    text = swapgb.synth_fasta(seed=k, genome_len=30_000, n_reads=6_000, read_len=100, sub_rate=0.01)
    _check(swapgb.Graph().build_reads(swapgb.Opts(k=k, cutoff=1), swapgb.reads_from_fasta(text, k)))


def test_more_than_the_radix_threshold():
    text = swapgb.synth_fasta(seed=3, genome_len=2_500_000, n_reads=100_000, read_len=100, sub_rate=0.0)
    for k in (19, 25, 31):
        g = swapgb.Graph().build_reads(swapgb.Opts(k=k, cutoff=1), swapgb.reads_from_fasta(text, k))
        assert g.size() > 1 << 20
        _check(g)


def test_batch_samples_of_several_k():
    texts = [swapgb.synth_fasta(seed=50 + i, genome_len=2_000 * (i + 1), n_reads=3_000, read_len=100, sub_rate=0.005)
             for i in range(4)]
    batch = [(swapgb.reads_from_fasta(t, k), k, 2) for t, k in zip(texts, (13, 21, 27, 20))]
    g = swapgb.Graph().build_batch(swapgb.Opts(), batch)
    for i in range(4):
        keys, mult = g.batch_copy_out(i, sorted=False)
        skeys, smult = g.batch_copy_out(i, sorted=True)
        order = np.argsort(keys)
        assert np.array_equal(skeys, keys[order]) and np.array_equal(smult, mult[order])
