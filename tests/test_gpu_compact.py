"""Unitig compaction by doubled successor tables at the path lengths where it can go wrong
(no 1-in-1-out node, one, and around the powers of two), at the word edges of the key, and
for a path whose first k bases equal its reverse complement's, against the oracle (sequences, edges and
coverages, as test_gpu_parity.compare_compaction compares them)."""
import pytest

from fastbact_gb300 import api
from test_gpu_parity import compare_compaction, rand_seqs

pytestmark = pytest.mark.gpu

COMP = bytes.maketrans(b"ACGT", b"TGCA")


@pytest.mark.parametrize("k,kb", [(3, 64), (21, 64), (31, 64), (32, 128), (33, 128), (63, 128), (64, 256), (77, 256), (96, 256),
                                  (97, 256), (127, 256)])
def test_path_lengths_and_hairpins(ctx, k, kb):
    nodes = [0, 1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 1000]
    seqs = [rand_seqs(100 + m, 1, k + 1 + m, k + 1 + m)[0] for m in nodes] if k > 11 else []
    stem, loop = rand_seqs(7, 1, 2 * k + 9, 2 * k + 9)[0], rand_seqs(8, 1, 2 * k + 3, 2 * k + 3)[0]
    seqs.append(stem + loop + stem[::-1].translate(COMP))   # the loop leaves a node and comes back to it from behind
    x, y, z = (rand_seqs(50 + i, 1, 2 * k + 5, 2 * k + 5)[0] for i in range(3))
    seqs += [x + y + z, rand_seqs(60, 1, 2 * k, 2 * k)[0] + y + rand_seqs(61, 1, 2 * k, 2 * k)[0]]  # a shared middle: branches
    reads = [s for s in seqs for _ in range(4)]
    bank = api.ReadBank(merged_reads=api.BitSeqArena.from_seqs(reads))
    compare_compaction(ctx, bank, k, kb, 16, None, 14)


@pytest.mark.parametrize("k,kb", [(5, 64), (20, 64), (21, 64), (31, 64), (32, 128), (33, 128), (64, 256), (77, 256), (127, 256)])
@pytest.mark.parametrize("extra", [1, 2, 3, 4, 5, 40, 301])
def test_palindromic_contigs(ctx, k, kb, extra):
    """A contig that is its own reverse complement passes every row twice: the walk stops at its
    middle, an edge (odd k) or a k-mer (even k) that is its own reverse complement."""
    x = rand_seqs(40 + extra, 1, k // 2 + extra, k // 2 + extra)[0]
    y = rand_seqs(3, 1, 3 * k, 3 * k)[0]
    for seqs in ([x + x[::-1].translate(COMP)], [x + x[::-1].translate(COMP), y]):
        if k == 5 and (extra > 4 or len(seqs) > 1):  # the short words meet: branches
            continue
        bank = api.ReadBank(merged_reads=api.BitSeqArena.from_seqs([s for s in seqs for _ in range(4)]))
        compare_compaction(ctx, bank, k, kb, 16, None, 14)


@pytest.mark.parametrize("k,kb", [(21, 64), (32, 128), (77, 256)])
def test_hairpin_on_a_branch(ctx, k, kb):
    """A palindromic path that leaves a branching node and comes back to it by the same edge."""
    a, b, x = (rand_seqs(70 + i, 1, 2 * k + i, 2 * k + i)[0] for i in range(3))
    stem = a + x
    seqs = [stem + stem[::-1].translate(COMP), a + b]
    bank = api.ReadBank(merged_reads=api.BitSeqArena.from_seqs([s for s in seqs for _ in range(4)]))
    compare_compaction(ctx, bank, k, kb, 16, None, 14)
