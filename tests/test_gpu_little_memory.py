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
