"""The merge and the passes over its lines at the sizes where their kernels
change over: the line sort (one block up to 1024 lines, splitters above), the
line scan (one block up to 16384), and the parts of 1024 bytes in which a
rewrite moves an arc's string. Everything is compared with the oracle exactly."""
import random

import pytest

import oracle
import swapgb

pytestmark = pytest.mark.gpu

K = 21


def _lines(text: bytes) -> list[bytes]:
    return sorted(l for l in text.split(b"\n") if l)


def _merged(text: bytes, k: int = K, cutoff: int = 2) -> swapgb.Graph:
    g = swapgb.Graph()
    g.build_fasta(swapgb.Opts(k=k, cutoff=cutoff), text)
    g.merge()
    keys, mult = oracle.records(text, k, cutoff)
    want = oracle.merge_text(keys, mult, k)
    got = g.merged_text()
    assert len(got) == len(want) and _lines(got) == _lines(want)
    firsts = [int(l.split(b" ", 1)[0]) for l in got.split(b"\n") if l]
    assert firsts == sorted(firsts)
    return g


@pytest.mark.parametrize("fragments", [1, 511, 512, 513, 8192, 8193])
def test_lines_of_fragments(fragments):
    """Separate fragments of a few bases more than k: two lines each."""
    rng = random.Random(fragments)
    text = ""
    for i in range(fragments):
        r = "".join(rng.choice("ACGT") for _ in range(K + 3 + i % 4))
        text += f">a{i}\n{r}\n>b{i}\n{r}\n"
    g = _merged(text.encode())
    assert g.merge_info()["nodes"] == 2 * fragments


@pytest.mark.parametrize("arc", [1, 1023, 1024, 1025, 2048, 2049, 3073, 40_000])
def test_rewritten_arcs(arc):
    """A sequence whose chain spells an arc of `arc` bases on one side of a
    branch, a tip: the tip goes, the line is rewritten, the branch merges."""
    rng = random.Random(arc)
    n = arc + K
    seq = "".join(rng.choice("ACGT") for _ in range(n + 60))
    at = n - K  # the branch's k-mer starts here: `arc` bases after the first
    other = seq[at:at + K] + ("A" if seq[at + K] != "A" else "C") + "".join(rng.choice("ACGT") for _ in range(5))
    reads = [seq[i:i + 100] for i in range(0, len(seq) - 99, 20)] + [seq[-100:], seq[:100]]
    reads = [r for r in reads for _ in range(6)] + [other] * 3
    text = "".join(f">r{i}\n{r}\n" for i, r in enumerate(reads)).encode()
    g = _merged(text)
    before = g.merged_text()
    g.remove_tips()
    tips = g.merged_text()
    want, _ = oracle.prune_text(before, K, oracle.PRUNE_TIPS, oracle.tips_last_order(before, K))
    assert _lines(tips) == _lines(want) and len(tips) == len(want)
    merged = g.simplify()
    want, n_merged = oracle.simplify_text(tips, K, oracle.lines_tree_order(tips, K))
    got = g.merged_text()
    assert merged == n_merged and _lines(got) == _lines(want) and len(got) == len(want)
