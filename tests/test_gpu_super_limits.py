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
