"""Unitig compaction by doubled successor tables at the path lengths where it can go wrong
(no 1-in-1-out node, one, and around the powers of two), at the word edges of the key, and
for a path whose first k bases equal its reverse complement's, against the oracle (sequences, edges and
coverages, as test_gpu_parity.compare_compaction compares them)."""
import ctypes as C

import numpy as np
import pytest

from fastbact_gb300 import _native as N
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


@pytest.mark.parametrize("k,kb", [(31, 64), (77, 256)])
def test_less_memory_than_tables(k, kb):
    """A pool with room for some of the tables, for one, and for none: the same unitigs from
    fewer of them, an isolated cycle (whose tables never run out) among them."""
    x, line, ring = (rand_seqs(90 + i, 1, n, n)[0] for i, n in enumerate((3000, 60_000, 40_000)))
    pal = x + x[::-1].translate(COMP)
    seqs = [s[i:i + 250] for s in (line, ring + ring[:300], pal) for i in range(0, len(s) - 249, 25)] + [line[-300:], pal[:300]] * 2
    seqs += [rand_seqs(200 + m, 1, k + 1 + m, k + 1 + m)[0] for m in (0, 1, 2, 7, 8, 9, 40)] * 4
    c = api.Context(0, pool_bytes=512 << 20)

    def largest():
        free, block = C.c_uint64(), C.c_uint64()
        N.check(N.lib().fbk_ctx_pool_free(c.handle, C.byref(free), C.byref(block)), c.handle)
        return block.value

    try:
        bank = api.ReadBank(merged_reads=api.BitSeqArena.from_seqs(seqs))
        table = api.build_cdbg_with_contigs_ext(bank, [], k, None, None, ctx=c, key_bits=kb, counter_bits=16, cms_log2_width=18)
        n = table.info()[1]
        seq, cov, circ, edges = api.compact(table)
        want = sorted(zip(seq, cov.tolist(), circ.tolist()))
        assert circ.sum() == 1 and max(map(len, seq)) > 50_000
        index = 4 * (1 << (2 * n - 1).bit_length())
        counts = []
        c.set_timing(True)
        for rest in (1 << 40, 120 * n, 60 * n, 32 * n, 22 * n, 12 * n):   # besides the index; the last holds no table
            fill, p = [], 18
            while p >= 4:                   # a sketch of 4 << p bytes at a time
                if largest() - (4 << p) >= index + rest:
                    fill.append(api.HyperLogLog(p, c))
                else:
                    p -= 1
            c.timing_reset()
            seq, cov, circ, edges = api.compact(table)
            counts.append(c.timing("compact_next")[1])
            assert sorted(zip(seq, cov.tolist(), circ.tolist())) == want
            for f in fill:
                f.release()
        assert counts[-1] == 0 and sorted(counts, reverse=True) == counts and len(set(counts)) > 3
    finally:
        c.close()
