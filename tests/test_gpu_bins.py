"""The build over minimizer bins at the sizes where it can go wrong, against the oracle:
the accumulator, the SolidKmerNode rows and the digest (integers, tolerance 0).

k = 17 is the smallest it takes; 31/32/33, 63/64/65 and 95/96/97 are the word edges of the
key; 127 the largest k.  The banks hold reads of exactly k and k + 1 bases among ordinary
ones (windows with no neighbour, with one, with two, of the same k-mers and of their reverse
complements), more distinct keys than a group's entries (windows put off to a later turn, and
a group taken in parts), groups of more than 65535 windows (wide counts), reads cut into
several runs, and reads that overlap in the packed words (left to the record buckets)."""
import ctypes as C

import numpy as np
import pytest

from fastbact_gb300 import _native as N
from fastbact_gb300 import api
from test_gpu_parity import compare_build, compare_gate_only, rand_seqs

pytestmark = pytest.mark.gpu

COMP = bytes.maketrans(b"ACGT", b"TGCA")
KS = [(17, 64), (21, 64), (31, 64), (32, 128), (33, 128), (63, 128), (64, 256), (65, 256), (95, 256), (96, 256), (97, 256),
      (127, 256)]


def rc(s):
    return s[::-1].translate(COMP)


def bank_of(seqs):
    a, b = len(seqs) // 3, 2 * len(seqs) // 3
    return api.ReadBank(api.BitSeqArena.from_seqs(seqs[:a]), api.BitSeqArena.from_seqs(seqs[a:b]), api.BitSeqArena.from_seqs(seqs[b:]))


def low_minimizer():
    """A 15-mer whose hash is below nearly every other's, so that it is the minimizer of
    every window that holds it (the hash of k_bin_runs)."""
    rng = np.random.default_rng(7)
    codes = rng.integers(0, 4, (1 << 20, 15)).astype(np.uint64)
    w = np.uint64(4) ** np.arange(15, dtype=np.uint64)
    rev = (3 - codes) @ w                   # base i at bits 2 i: the reverse complement's integer
    fwd = codes @ w[::-1]
    z = ((np.minimum(fwd, rev) ^ np.uint64(0x3C6EF372)) * np.uint64(0x9E3779B1)) & np.uint64(0xFFFFFFFF)
    z ^= z >> np.uint64(15)
    z = (z * np.uint64(0x85EBCA77)) & np.uint64(0xFFFFFFFF)
    return bytes(b"ACGT"[c] for c in codes[int(np.argmin(z))])


@pytest.mark.parametrize("k,kb", KS)
@pytest.mark.parametrize("acc_filter", [0, 1, 2])
def test_short_reads_and_word_edges(k, kb, acc_filter):
    rng = np.random.default_rng(k)
    genome = rand_seqs(int(rng.integers(1 << 30)), 1, 3000, 3000)[0]
    seqs = []
    for i in range(0, 2700, 7):
        seqs.append(genome[i:i + 290])
    for i in range(0, 2700, 11):  # one window, two windows, both strands; some seen only here
        seqs += [genome[i:i + k], rc(genome[i + 3:i + 3 + k + 1]), rc(genome[i:i + k])]
    seqs += rand_seqs(5, 40, k, k) + rand_seqs(6, 40, k + 1, k + 2) + rand_seqs(8, 20, 1, k - 1) + [b"", b"A" * 400, b"AC" * 150]
    lone = rand_seqs(9, 30, k + 2, k + 2)   # a window without neighbours, then the same k-mer with both
    seqs += [s[1:-1] for s in lone] + lone
    order = rng.permutation(len(seqs))
    c = api.Context(0)
    try:
        c.set_tuning(acc_filter=acc_filter)
        compare_gate_only(c, bank_of([seqs[i] for i in order]), k, kb, 16, None, 12)
        compare_gate_only(c, bank_of([seqs[i] for i in order]), k, kb, 4, 2, 14)
    finally:
        c.close()


@pytest.mark.parametrize("k,kb", [(21, 64), (31, 64), (45, 128), (77, 256)])
def test_more_keys_than_a_group_holds(ctx, k, kb):
    """All keys distinct (put off to later turns), then 20,000 windows of one minimizer (taken
    in parts), some of them twice."""
    seqs = rand_seqs(3, 700, 100, 400)
    compare_gate_only(ctx, bank_of(seqs), k, kb, 16, None, 14)
    x = low_minimizer()
    flank = rand_seqs(4, 2400, 60, 80)
    seqs = [flank[i] + x + flank[i + 1] for i in range(0, 2400, 2)]
    seqs += [rc(s) for s in seqs[::9]] + [s[5:] for s in seqs[::7]]
    compare_gate_only(ctx, bank_of(seqs), k, kb, 16, None, 16)


@pytest.mark.parametrize("k,kb", [(21, 64), (55, 128), (99, 256)])
def test_groups_with_wide_counts(ctx, k, kb):
    """One k-mer 100,000 times and more (its counts pass 65535), with reads of several
    thousand bases (runs cut every 2048 windows) and ordinary ones around it."""
    seqs = [b"A" * 3000] * 30 + [b"T" * 2500] * 20 + [b"ACG" * 900] * 50 + rand_seqs(11, 200, 150, 300)
    compare_gate_only(ctx, bank_of(seqs), k, kb, 16, None, 12)


@pytest.mark.parametrize("k", [21, 33, 77])
def test_sampled_sizes(ctx, k):
    """Above 4 M windows a sample of the bins sizes the groups and the rows."""
    p = api.synth_params(seed=91, genome_len=150_000, coverage=60.0, sub_rate=0.008, n_repeats=3, repeat_len=900)
    bank = api.synth_isolate(p, threads=0, sample_pairs=0)[0]
    assert sum(int(np.maximum(a.lengths.astype(np.int64) - k + 1, 0).sum()) for a in bank.arenas) > 4 << 20
    compare_gate_only(ctx, bank, k, api.key_bits_for_k(k), 16, None, 18)


@pytest.mark.parametrize("k,kb", [(17, 64), (31, 64), (32, 128), (63, 128), (77, 256), (99, 256), (127, 256)])
@pytest.mark.parametrize("acc_filter", [0, 2])
def test_kept_sketch(k, kb, acc_filter):
    """A build that returns its sketch: every counter, and the rows that it gates, with windows
    that have a neighbour on one side or none, counts beyond 65535 and keys of every fate; and
    a second build on that sketch (its distinct count sizes the table)."""
    seqs = rand_seqs(31, 300, k, 3 * k) + rand_seqs(32, 60, k, k + 1) + [b"A" * 3000] * 25 + [b"T" * 900] * 3 + [b"ACG" * 900] * 50
    seqs += [rc(s) for s in seqs[::3]] + [s[1:] for s in seqs[:300:4]] + [s[:-2] for s in seqs[:300:5]] + seqs[:60]
    bank = bank_of([seqs[i] for i in np.random.default_rng(k).permutation(len(seqs))])
    caps = []
    for form in (1, 0):
        c = api.Context(0)
        try:
            c.set_tuning(acc_filter=acc_filter, build_form=form)
            for cb, log2w in ((16, 16), (4, 10)):
                compare_build(c, bank, k, kb, cb, None, log2w)
            d = api.DeviceBank(c, bank)
            _, cms = api.build_cdbg_with_contigs_ext(d, [], k, None, None, ctx=c, key_bits=kb, counter_bits=16, cms_log2_width=16, keep_cms=True)
            t = api.solid_build(c, d, cms, k)
            caps.append((t.info(), t.digest()))
        finally:
            c.close()
    assert caps[0] == caps[1]


def test_overlapping_reads():
    """Reads that share packed words: adjacent windows of the bank need not be a read's.
    (Every accumulated key is kept: which ones a filter keeps is the form's own.)"""
    ctx = api.Context(0)
    ctx.set_tuning(acc_filter=0)
    a = api.BitSeqArena.from_seqs(rand_seqs(21, 1, 4000, 4000))
    offs = np.array([0, 50, 50, 70, 100, 60, 3000, 2990], np.uint64)
    lens = np.array([80, 100, 100, 31, 300, 40, 200, 220], np.uint32)
    seq = a.extract_ascii(0)
    shared = api.ReadBank(api.BitSeqArena(a.data, offs, lens), api.BitSeqArena(), api.BitSeqArena())
    apart = api.ReadBank(api.BitSeqArena.from_seqs([seq[int(o):int(o + n)] for o, n in zip(offs, lens)]))
    got = []
    for bank in (shared, apart):
        t = api.build_cdbg_ext(bank, 31, 1, 100000, ctx=ctx, counter_bits=4, cms_log2_width=12)
        u = api.build_cdbg_ext(bank, 31, None, 100000, ctx=ctx, counter_bits=4, cms_log2_width=12)
        got.append((t.digest(), t.pushes(), u.digest(), u.pushes(), u.acc_digest()))
        t.release()
        u.release()
    ctx.close()
    assert got[0] == got[1]


def one_fold(n, seed=5):
    """n reads, twice each, whose first 63-mers share their minimizer and the fold of their two
    words, which is all that any hash of a key sees."""
    rng = np.random.default_rng(seed)
    code = np.zeros(256, np.uint8)
    code[list(b"ACGT")] = range(4)
    x = code[np.frombuffer(low_minimizer(), np.uint8)]
    w0 = rng.integers(0, 4, (n, 31)).astype(np.uint8)
    w0[:, 0] = 0                            # with the last base below: smaller than their reverse complements
    w0[:, 16:31] = x
    c = rng.integers(0, 4, 32).astype(np.uint8)
    c[31] = x[14]
    w1 = np.concatenate([np.zeros((n, 1), np.uint8), w0], 1) ^ c
    reads = np.concatenate([w0, w1, rng.integers(0, 4, (n, 1)).astype(np.uint8)], 1)
    return [bytes(r) for r in np.frombuffer(b"ACGT", np.uint8)[reads]] * 2


def uneven_reads(seed, genome_len, n, length, long_ones, rate=0.002):
    """n reads of about `length` bases and a few long ones, from a genome, with errors."""
    rng = np.random.default_rng(seed)
    g = np.frombuffer(rand_seqs(seed, 1, genome_len, genome_len)[0], np.uint8)
    lens = list(rng.integers(length - length // 8, length + length // 8, n))
    for L in long_ones:
        lens.insert(int(rng.integers(len(lens))), L)
    out = []
    for L in lens:
        a = int(rng.integers(0, genome_len - L + 1))
        r = g[a:a + L].copy()
        e = rng.random(L) < rate
        r[e] = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, int(e.sum()))]
        out.append(rc(r.tobytes()) if rng.random() < 0.5 else r.tobytes())
    return out


@pytest.mark.parametrize("k", [21, 31, 77])
@pytest.mark.parametrize("keep", [False, True])
@pytest.mark.parametrize("n,length,long_ones,binned", [(640, 7200, (150_000, 90_000), True), (8000, 620, (1_000_000,), False)])
def test_reads_of_uneven_length(k, keep, n, length, long_ones, binned):
    """A warp of k_bin_runs meets reads of many times the mean length: its log is too short and
    the runs are logged again with room for it, or, where that would take the logs of thousands
    of warps to the length of one, the build goes over the record buckets."""
    c = api.Context(0)
    try:
        seqs = uneven_reads(k, 1_200_000, n, length, long_ones)
        assert sum(len(s) - k + 1 for s in seqs) > 4 << 20
        c.set_timing(True)
        (compare_build if keep else compare_gate_only)(c, bank_of(seqs), k, api.key_bits_for_k(k), 16, None, 20)
        assert c.timing("bins_runs")[1] == (2 if binned else 1)
        assert (c.timing("bins_aggregate")[0] > 0) == binned and (c.timing("pass2_emit")[0] > 0) != binned
    finally:
        c.close()


@pytest.mark.parametrize("k", [21, 77])
@pytest.mark.parametrize("share", [0.02, 0.1])
def test_frequent_kmer(ctx, k, share):
    """One k-mer many times a group's windows, among more than 4 M ordinary ones: its bin has a
    group of its own, between those of the bins before and after it."""
    seqs = uneven_reads(k, 150_000, 36_000, 200, (), 0.004)
    n = int(share * len(seqs))
    seqs[100:100 + n] = [b"G" * len(s) for s in seqs[100:100 + n]]
    seqs[200:200 + n // 8] = [s[:30] + s[30:31].replace(b"G", b"T") + s[31:] for s in seqs[200:200 + n // 8]]
    assert sum(len(s) - k + 1 for s in seqs) > 4 << 20
    compare_gate_only(ctx, bank_of(seqs), k, api.key_bits_for_k(k), 16, None, 18)


@pytest.mark.parametrize("keep", [False, True])
def test_keys_of_one_fold(keep):
    """14,000 keys that no hash tells apart: a group of them cannot be taken in parts, and the
    build goes over the record buckets."""
    c = api.Context(0)
    try:
        c.set_timing(True)
        (compare_build if keep else compare_gate_only)(c, bank_of(one_fold(14_000) + rand_seqs(9, 100, 80, 200)), 63, 128, 16, None, 18)
        assert c.timing("bins_aggregate")[1] == 1 and c.timing("pass2_emit")[1] > 0
    finally:
        c.close()


def test_record_options_and_the_form():
    """An option of the record buckets takes the builds there, which build_form tells and undoes."""
    c = api.Context(0)
    try:
        bank = bank_of(rand_seqs(1, 50, 100, 200) * 2)

        def binned():
            c.timing_reset()
            c.set_timing(True)
            api.build_cdbg_ext(bank, 31, None, 10_000, ctx=c, counter_bits=16, cms_log2_width=12).release()
            return c.timing("bins_aggregate")[0] > 0

        assert c.get_tuning("build_form") == 1 and binned()
        c.set_tuning(bucket_bytes=c.get_tuning("bucket_bytes"))
        assert c.get_tuning("build_form") == 0 and not binned()
        c.set_tuning(build_form=1)
        assert c.get_tuning("build_form") == 1 and binned()
        c.set_tuning(build_form=0)
        assert c.get_tuning("build_form") == 0 and not binned()
    finally:
        c.close()


@pytest.mark.parametrize("option", [dict(build_form=0), dict(load_factor=0.5), {}])
def test_a_fork_builds_in_its_parents_form(option):
    c = api.Context(0)
    h = C.c_void_p()
    try:
        c.set_tuning(**option)
        N.check(N.lib().fbk_ctx_fork(c.handle, C.byref(h)), c.handle, "fork")
        v = C.c_double()
        N.check(N.lib().fbk_ctx_get_tuning(h, b"build_form", C.byref(v)), h, "get_tuning")
        assert v.value == c.get_tuning("build_form") == (0 if option else 1)
    finally:
        N.lib().fbk_ctx_destroy(h)
        c.close()


def at_rich_reads(seed, genome_len, n, gc):
    """150-base reads of a genome whose few frequent words are the minimizers of many k-mers, with
    tracts of one base and errors."""
    rng = np.random.default_rng(seed)
    g = rng.choice(np.frombuffer(b"ACGT", np.uint8), genome_len, p=[(1 - gc) / 2, gc / 2, gc / 2, (1 - gc) / 2])
    for a in rng.integers(0, genome_len - 40, genome_len // 400):
        g[a:a + int(rng.integers(8, 30))] = ord("A")
    out = []
    for a in rng.integers(0, genome_len - 150, n):
        r = g[a:a + 150].copy()
        r[rng.random(150) < 0.004] = ord("C")
        out.append(rc(r.tobytes()) if rng.random() < 0.5 else r.tobytes())
    return out


@pytest.mark.parametrize("k", [17, 21, 33, 77, 99])
@pytest.mark.parametrize("keep,genome_len,n", [(False, 80_000, 16_000), (True, 80_000, 16_000), (False, 300_000, 70_000)])
def test_frequent_minimizers(k, keep, genome_len, n):
    """Bins of many keys, scattered again over sub-bins, with and without a sample of the bins."""
    seqs = at_rich_reads(k, genome_len, n, 0.08) + [b"G" * 150] * 300 + [b"AC" * 75] * 300
    c = api.Context(0)
    try:
        c.set_timing(True)
        (compare_build if keep else compare_gate_only)(c, bank_of(seqs), k, api.key_bits_for_k(k), 16, None, 18)
        assert c.timing("bins_heavy")[1] == 5 and c.timing("bins_aggregate")[1] >= 1 and c.timing("pass2")[1] == 0
    finally:
        c.close()


@pytest.mark.parametrize("k,keep,acc_filter", [(31, False, 0), (31, True, 1), (77, False, 1), (31, False, 2), (127, True, 2)])
def test_short_of_memory(k, keep, acc_filter):
    """Pools of every size between too small and ample: what the record buckets build is built,
    whether the bins find their memory, in part of their steps or not at all."""
    bank = bank_of(uneven_reads(k, 100_000, 32_000, 120 + k, (), 0.004))
    got = {}
    for mb in (16, 48, 64, 80, 96, 112, 128, 144, 160, 176, 192, 208, 224, 256, 320, 448, 1024):
        for form in (0, 1):
            c = api.Context(0, pool_bytes=mb << 20)
            try:
                c.set_tuning(build_form=form, acc_filter=acc_filter)
                c.set_timing(True)
                t, cms = api.build_cdbg_with_contigs_ext(bank, [], k, None, None, ctx=c, counter_bits=16, cms_log2_width=20, keep_cms=True) if keep \
                    else (api.build_cdbg_ext(bank, k, None, 100_000, ctx=c, counter_bits=16, cms_log2_width=20), None)
                got[mb, form] = (t.info()[1], t.digest(), t.pushes(), cms.export().tobytes() if keep else None)
                got[mb, "route"] = (c.timing("bins_aggregate")[1] > 0, c.timing("pass2")[1] > 0)
            except N.FbkError as e:
                assert N.STATUS_NAMES[e.status] == "FBK_ERR_OOM", e
                got[mb, form] = None
            finally:
                c.close()
        if got[mb, 0] is not None or got[mb, 1] is not None:
            assert got[mb, 1] == (got[mb, 0] or got[mb, 1])
    done = {v for key, v in got.items() if key[1] in (0, 1)}
    assert len(done - {None}) == 1 and None in done
    routes = [v for key, v in got.items() if key[1] == "route"]
    assert routes[0] == (False, True) and routes[-1] == (True, False)


@pytest.mark.parametrize("k", [63, 77])
@pytest.mark.parametrize("keep", [False, True])
@pytest.mark.parametrize("acc_filter", [0, 2])
def test_a_sample_that_tells_too_little(k, keep, acc_filter):
    """Many distinct keys in one bin that is no part of the sample: the rows do not suffice, and
    the keys are counted again with the counted sizes."""
    x = low_minimizer()
    flank = rand_seqs(4, 16_000, k - 17, k - 15)
    seqs = uneven_reads(k, 20_000, 30_000, 230, (), 0.0) + [flank[i] + x + flank[i + 1] for i in range(0, 16_000, 2)] * 2
    assert sum(max(0, len(s) - k + 1) for s in seqs) > 4 << 20
    c = api.Context(0)
    try:
        c.set_tuning(acc_filter=acc_filter)
        c.set_timing(True)
        (compare_build if keep else compare_gate_only)(c, bank_of(seqs), k, api.key_bits_for_k(k), 16, None, 20)
        # (filtered, the keys seen twice are only listed for the sketch, and not at all for one that is kept)
        assert c.timing("bins_aggregate")[1] == (1 if keep and acc_filter else 2) and c.timing("pass2")[1] == 0
    finally:
        c.close()


@pytest.mark.parametrize("k,kb,filtered", [(21, 64, True), (55, 128, True), (21, 64, False)])
def test_small_builds_filter_as_larger_ones(k, kb, filtered):
    """Below the sample's size too, a build whose distinct keys exceed a fifth of its windows keeps
    out of the accumulator what cannot become solid."""
    seqs = uneven_reads(k, 400_000 if filtered else 8_000, 3_000, 200, (), 0.002)
    c = api.Context(0)
    try:
        compare_gate_only(c, bank_of(seqs), k, kb, 16, None, 16)
        compare_build(c, bank_of(seqs), k, kb, 16, None, 16)
        info = []
        for acc_filter in (1, 0):
            c.set_tuning(acc_filter=acc_filter)
            t = api.build_cdbg_ext(bank_of(seqs), k, None, 100_000, ctx=c, counter_bits=16, cms_log2_width=16)
            info.append((t.filtered(), *t.info()[:2], t.pushes()))
        assert info[0][0] == filtered and not info[1][0] and info[0][2:] == info[1][2:]
        assert (info[0][1] < info[1][1]) == filtered
    finally:
        c.close()


@pytest.mark.parametrize("k", [21, 77])
@pytest.mark.parametrize("genome_len,acc_filter", [(3_000, 0), (20_000, 1), (700, 2)])
def test_deep_banks(k, genome_len, acc_filter):
    """Depths of hundreds to ten thousand: every bin that holds anything holds many windows, few of
    them distinct, and is sampled by a part of its keys."""
    seqs = uneven_reads(k, genome_len, 60_000, 130 + k // 2, (), 0.004)
    c = api.Context(0)
    try:
        c.set_tuning(acc_filter=acc_filter)
        c.set_timing(True)
        compare_gate_only(c, bank_of(seqs), k, api.key_bits_for_k(k), 16, None, 18)
        assert c.timing("bins_sample")[1] == 1 and c.timing("bins_aggregate")[1] == 1 and c.timing("pass2")[1] == 0
    finally:
        c.close()


@pytest.mark.parametrize("k,rate,keep,binned", [(77, 0.06, False, False), (127, 0.04, True, False), (77, 0.002, False, True), (33, 0.15, False, True)])
def test_banks_of_mostly_new_keys(k, rate, keep, binned):
    """Wide keys of which most occur once go over the record buckets once a sample says so."""
    seqs = uneven_reads(k, 600_000, 34_000, 130 + k, (), rate)
    c = api.Context(0)
    try:
        c.set_timing(True)
        (compare_build if keep else compare_gate_only)(c, bank_of(seqs), k, api.key_bits_for_k(k), 16, None, 20)
        assert c.timing("bins_sample")[1] == 1 and (c.timing("bins_aggregate")[1] > 0) == binned and (c.timing("pass2")[1] > 0) != binned
    finally:
        c.close()
