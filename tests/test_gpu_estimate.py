"""The estimator's sample loop where its rounds and forms can go wrong, against the oracle's
sequential loop: registers and whole numbers, and the floats from the same operations
(tolerance 0).

The loop stops at the first checkpoint, in a later round, at no checkpoint (the sample ends
inside a segment), or has fewer pairs than one; small sketches, whose counters are shared by
many k-mers; every word count of k; and a sample whose reads do not lie in read order in
its packed words.  Samples of more than 8 M k-mers go over the distinct ones (k of every word
count, counters shared by several k-mers, a round that begins in the middle), unless most of
them are distinct."""
import numpy as np
import pytest

from fastbact_gb300 import api
from oracle import orc
from test_gpu_bins import at_rich_reads, uneven_reads
from test_gpu_parity import sample_reads

pytestmark = pytest.mark.gpu


def same(ctx, sample, n, stats, k, p, log2w):
    rc, oe, ort, ors = orc.estimate_from_reads(sample_reads(sample, n), orc.count_stats(**stats.__dict__), 250000, 50.0, k=k,
                                               cms_width=1 << log2w, hll_p=p)
    assert rc == 0
    ge, rt, rs = api.estimate_sample(ctx, sample, n, stats, max_pairs=250000, target_cov=50.0, k=k, hll_p=p, cms_log2_width=log2w)
    assert np.array_equal(rt, ort) and np.array_equal(rs, ors)
    for f in ("genome_size", "estimated_cov", "subsample_factor", "u_ge_1", "u_ge_2", "sample_kmer_depth", "pairs_sampled", "m_sample"):
        assert getattr(ge, f) == getattr(oe, f), f
    return ge.pairs_sampled


@pytest.mark.parametrize("genome,cov,k,p,log2w", [
    (20_000, 120.0, 21, 14, 23), (150_000, 30.0, 21, 14, 23), (150_000, 60.0, 31, 16, 16), (300_000, 25.0, 17, 14, 20),
    (300_000, 25.0, 11, 12, 12), (40_000, 25.0, 33, 14, 18), (200_000, 40.0, 127, 14, 20), (100_000, 90.0, 64, 4, 14)])
@pytest.mark.parametrize("in_order", [True, False])
def test_sample_loop_rounds(ctx, genome, cov, k, p, log2w, in_order):
    prm = api.synth_params(seed=genome + k, genome_len=genome, coverage=cov, gc=0.5, n_repeats=3, repeat_len=1500, sub_rate=0.005)
    _, _, sample, n, stats = api.synth_isolate(prm, sample_pairs=150_000)
    if not in_order:
        sample = api.BitSeqArena(sample.data, sample.offsets[::-1].copy(), sample.lengths[::-1].copy())
    same(ctx, sample, n, stats, k, p, log2w)


@pytest.mark.parametrize("genome,cov,k,p,log2w,errors,distinct", [
    (2_500_000, 5.0, 21, 14, 23, 0.005, True), (2_500_000, 5.0, 31, 14, 20, 0.005, True), (2_000_000, 6.0, 33, 16, 23, 0.002, True),
    (1_000_000, 19.0, 77, 14, 16, 0.001, True), (1_000_000, 27.0, 101, 14, 22, 0.001, True), (2_000_000, 10.0, 77, 14, 23, 0.03, False)])
def test_whole_samples(ctx, genome, cov, k, p, log2w, errors, distinct):
    prm = api.synth_params(seed=genome + k, genome_len=genome, coverage=cov, gc=0.5, n_repeats=5, repeat_len=2000, sub_rate=errors)
    _, _, sample, n, stats = api.synth_isolate(prm, sample_pairs=150_000)
    assert int(np.maximum(sample.lengths[:2 * n].astype(np.int64) - k + 1, 0).sum()) > 8 << 20
    ctx.timing_reset()
    ctx.set_timing(True)
    same(ctx, sample, n, stats, k, p, log2w)
    ctx.set_timing(False)
    assert (ctx.timing("est_first_regs")[0] > 0) == distinct


@pytest.mark.parametrize("k", [21, 31])
@pytest.mark.parametrize("long_ones,runs", [((120_000, 80_000), 2), ((1_000_000, 7_500), 1)])
def test_samples_of_uneven_length(ctx, k, long_ones, runs):
    """Reads of many times the mean length: the runs of one warp do not fit its log, which is
    made longer, or the sample goes over its occurrences."""
    seqs = uneven_reads(k, 1_200_000, 1400, 7500, long_ones)
    sample = api.BitSeqArena.from_seqs(seqs)
    n = len(seqs) // 2
    lens = [len(s) for s in seqs]
    stats = api.ExactCountStats(n, sum(lens[::2]), sum(lens[1::2]), sum(lens), min(lens), max(lens), float(np.mean(lens)), int(np.median(lens)))
    assert sum(len(s) - k + 1 for s in seqs) > 8 << 20
    ctx.timing_reset()
    ctx.set_timing(True)
    same(ctx, sample, n, stats, k, 14, 20)
    ctx.set_timing(False)
    assert ctx.timing("est_runs")[1] == runs
    assert (ctx.timing("est_first_keys")[0] > 0) == (runs == 2)


@pytest.mark.parametrize("n,length", [(1400, 7500), (70_000, 150)])
def test_keys_met_by_many_warps_at_once(ctx, n, length):
    """Deep samples, whose k-mers are entered several times before the first entry is seen: the
    distinct ones find room all the same."""
    seqs = uneven_reads(n, 1_200_000, n, length, ())
    sample = api.BitSeqArena.from_seqs(seqs)
    lens = [len(s) for s in seqs]
    stats = api.ExactCountStats(n // 2, sum(lens[::2]), sum(lens[1::2]), sum(lens), min(lens), max(lens), float(np.mean(lens)),
                                int(np.median(lens)))
    ctx.timing_reset()
    ctx.set_timing(True)
    same(ctx, sample, n // 2, stats, 21, 14, 20)
    ctx.set_timing(False)
    assert ctx.timing("est_first_keys")[1] == ctx.timing("est_first_regs")[1] > 0


@pytest.mark.parametrize("genome,longest,rounds", [(100_000, 20_000, 1), (600_000, 20_000, 1), (600_000, 10_000, 2)])
def test_long_reads_in_one_round(ctx, genome, longest, rounds):
    """A sample with a long read is taken at once, whether the loop stops at its first checkpoint
    or at its end."""
    seqs = uneven_reads(genome, genome, 16_000, 400, (longest, 300))
    sample = api.BitSeqArena.from_seqs(seqs)
    n, lens = len(seqs) // 2, [len(s) for s in seqs]
    stats = api.ExactCountStats(n, sum(lens[::2]), sum(lens[1::2]), sum(lens), min(lens), max(lens), float(np.mean(lens)), int(np.median(lens)))
    ctx.timing_reset()
    ctx.set_timing(True)
    assert same(ctx, sample, n, stats, 21, 14, 18) == (6000 if genome == 100_000 else n)
    ctx.set_timing(False)
    assert ctx.timing("est_firstpos")[1] == rounds


@pytest.mark.parametrize("k", [21, 33])
def test_frequent_minimizers(ctx, k):
    """A sample of more than 8 M k-mers whose bins hold many keys each."""
    seqs = at_rich_reads(k, 1_000_000, 80_000, 0.1)
    sample = api.BitSeqArena.from_seqs(seqs)
    lens = [len(s) for s in seqs]
    stats = api.ExactCountStats(len(seqs) // 2, sum(lens[::2]), sum(lens[1::2]), sum(lens), min(lens), max(lens), 150.0, 150)
    ctx.timing_reset()
    ctx.set_timing(True)
    same(ctx, sample, len(seqs) // 2, stats, k, 14, 20)
    ctx.set_timing(False)
    assert ctx.timing("est_heavy")[1] >= 5 and ctx.timing("est_first_regs")[1] >= 1
