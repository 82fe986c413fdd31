"""The multi-k input filter at the edges of its rules, against the oracle's restatement (bytes,
tolerance 0): unitigs shorter than k, of k bases, at the window and length limits, empty, linear,
circular and branching on either side, lower case and N; k above and below 31; reads shorter than
k; pairs without a mate; no unitigs at all."""
import numpy as np
import pytest

from fastbact_gb300 import api
from oracle import orc
from test_gpu_parity import rand_seqs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph_k", [1, 15, 31, 45])
def test_window_rules(ctx, graph_k):
    rng = np.random.default_rng(graph_k)
    lens = [0, 1, 14, 15, 30, 31, 32, 349, 350, 351, 380, 381, 1999, 2000, 2001, 2030, 5000, 2000, 2600, 3000, 4000]
    seqs = [rand_seqs(100 + i, 1, n, n, b"ACGTACGTACGTacgtN")[0] for i, n in enumerate(lens)]
    circular = np.array([i in (8, 18) for i in range(len(lens))], np.uint8)
    # (from, side, to, reverse, overlap, support): unitig 19 branches on one side, 20 on the other, 16 has one edge a side
    edges = np.array([[19, 0, 1, 0, 5, 1], [19, 0, 2, 0, 5, 1], [20, 1, 3, 0, 5, 1], [20, 1, 4, 1, 5, 1], [16, 0, 5, 0, 5, 1],
                      [16, 1, 6, 0, 5, 1]], np.uint32)

    def reads(n):
        out = []
        for _ in range(n):
            s = seqs[int(rng.integers(len(seqs)))]
            a, m = int(rng.integers(0, len(s) + 1)), int(rng.choice([3, 14, 15, 16, 30, 31, 32, 44, 45, 46, 100, 150]))
            r = s[a:a + m] if rng.random() < 0.8 else rand_seqs(int(rng.integers(1 << 30)), 1, m, m)[0]
            out.append(r.upper().replace(b"N", b"A") or b"A")
        return out

    bank = api.ReadBank(*(api.BitSeqArena.from_seqs(reads(n)) for n in (300, 203, 200)))
    keep, kept = api.filter_active_reads(ctx, bank, seqs, circular, edges, graph_k)
    expected = orc.filter_active_reads(bank, seqs, circular, edges, graph_k)
    assert np.array_equal(keep, expected) and kept == int(expected.sum())
    keep, kept = api.filter_active_reads(ctx, bank, [], [], np.zeros((0, 6), np.uint32), graph_k)
    assert not keep.any() and kept == 0
