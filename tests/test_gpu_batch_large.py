"""A batch whose large isolates are built on their own, over minimizer bins, and whose small
ones share waves: every result field and row equals the single-isolate calls' and those of a
batch that takes all of them through the waves (integers, tolerance 0)."""
import numpy as np
import pytest

from fastbact_gb300 import api
from test_gpu_batch import POLICY, check_same, run_batch, single
from test_gpu_bins import one_fold

pytestmark = pytest.mark.gpu

# depth, genome: above 8 M k-mers, below, above and subsampled to 110x, subsampled below it
SPECS = [(130_000, 90.0), (40_000, 30.0), (110_000, 200.0), (60_000, 190.0)]


@pytest.mark.parametrize("kw", [dict(), dict(use_graphs=0, autotune=0), dict(max_wave=1), dict(max_wave_bytes=1 << 30)])
def test_large_and_small_isolates(ctx, kw):
    isolates = []
    for i, (g, cov) in enumerate(SPECS):
        isolates.append(api.synth_isolate(api.synth_params(seed=2000 + i, genome_len=g, coverage=cov), sample_pairs=150_000))
    expected = [single(ctx, iso) for iso in isolates]
    assert [e["factor"] < 1 for e in expected] == [False, False, True, True]
    got, _ = run_batch(ctx, isolates, **kw)
    check_same(got, expected)
    c = api.Context(0)
    try:
        c.set_tuning(build_form=0)
        waves, st = run_batch(c, isolates, **kw)
    finally:
        c.close()
    for a, b in zip(got, waves):
        for f in ("state", "subsample_reason", "fallback", "subsample_factor", "n_solid", "digest", "pushes", "kmers", "status"):
            assert getattr(a["res"], f) == getattr(b["res"], f), f
    assert st.isolates_done == len(SPECS)


def test_an_isolate_that_the_bins_decline():
    """A large isolate with keys that no hash tells apart goes to the waves alone: the others of
    the batch are done, and every field equals that of a batch without bins."""
    isolates = [api.synth_isolate(api.synth_params(seed=2100 + i, genome_len=g, coverage=140.0), sample_pairs=150_000)
                for i, g in enumerate((130_000, 140_000, 20_000))]
    bank = isolates[0][0]
    m, extra = bank.merged_reads, api.BitSeqArena.from_seqs(one_fold(14_000))
    bank.merged_reads = api.BitSeqArena(np.concatenate([m.data, extra.data]), np.concatenate([m.offsets, extra.offsets + np.uint64(32 * len(m.data))]),
                                        np.concatenate([m.lengths, extra.lengths]), np.concatenate([m.pair_idx, np.full(len(extra), m.pair_idx[-1])]))
    got = []
    for form in (1, 0):
        c = api.Context(0)
        try:
            c.set_tuning(build_form=form)
            c.set_timing(True)
            got.append(run_batch(c, isolates, k=63, key_bits=128)[0])
            assert c.timing("bins_aggregate")[1] == 2 * form
        finally:
            c.close()
    for a, b in zip(*got):
        for f in ("state", "subsample_reason", "fallback", "subsample_factor", "n_solid", "digest", "pushes", "kmers", "status"):
            assert getattr(a["res"], f) == getattr(b["res"], f), f
        assert a["res"].state == 3 and a["digest"] == b["digest"]
