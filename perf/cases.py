"""Timed cases of the k-mer counting front end: what an assembly pipeline has this
framework do for one isolate after another, through its public entry points.

A pipeline ingests a FASTQ pair, estimates the genome, builds the solid k-mer table
at each k of its ladder, compacts every table into unitigs, drops the reads that no
longer matter for the next k, and hands the rows on; cohorts go through batches.
Sizes come from fastbact_gb300/workloads.py and cohort.py (1 Mbp at 50x, 5 Mbp at
100x with k = 21/33/55/77, the 12 Mbp stress genome with k = 127, cohorts of uneven
depth) and reach down to plasmid-sized inputs, where launches and host turnarounds
are all there is.  Reads are the generator's (PE150, Phred tail decay, trimmed and
merged), so every seed is another genome with other errors.
"""
import math
import os
import tempfile

import numpy as np
import torch

from fastbact_gb300 import api

POLICY = dict(enable_auto_subsample=True, depth=110.0, threshold_ratio=150.0 / 110.0)
MAX_PAIRS, TARGET_COV, SAMPLE_PAIRS = 250_000, 110.0, 150_000
READ_LEN = 150

_ctx = None


def context():
    """The process's device context with its memory pool, as bench.py makes it."""
    global _ctx
    if _ctx is None:
        _ctx = api.Context(0, pool_bytes=60 << 30)
    return _ctx


def _case(name, kind, genome, cov, k=31, sub=0.005, gc=0.5, cb=16, log2w=0, tsc=0, repeats=0, isolates=1, hll_p=14):
    """tsc 0: the default solid threshold; log2w 0: the sketch sized from the genome size."""
    return dict(name=name, kind=kind, genome=genome, cov=cov, k=k, sub=sub, gc=gc, cb=cb, log2w=log2w, tsc=tsc,
                repeats=repeats, isolates=isolates, hll_p=hll_p)


def listed():
    return [
        # a plasmid or amplicon at low depth: launches, allocations and host turnarounds
        _case("build_20kb_30x_k31", "build", 20_000, 30.0, cb=4),
        # the reference's own CPU case: 1 Mbp, 50x, k = 31
        _case("build_1mbp_50x_k31", "build", 1_000_000, 50.0, log2w=22),
        # a middle genome at an odd size, the second k of the ladder (128-bit keys), the reference's nibble counters
        _case("build_2.3mbp_41x_k33", "build", 2_345_677, 41.0, k=33, gc=0.38, cb=4),
        # isolate scale: first and last k of the benchmark's ladder (64- and 256-bit keys)
        _case("build_5mbp_100x_k21", "build", 5_000_000, 100.0, k=21, gc=0.51, log2w=24, repeats=7),
        _case("build_5mbp_100x_k77", "build", 5_000_000, 100.0, k=77, gc=0.51, log2w=24, repeats=7),
        # the stress genome's k and error rate: the widest keys, few windows per read
        _case("build_6mbp_60x_k127", "build", 6_000_000, 60.0, k=127, sub=0.01, gc=0.66, log2w=26, repeats=10),
        # a caller that keeps the pass-1 sketch (merging ranks' sketches, re-gating later)
        _case("build_sketch_1mbp_50x_k31", "sketch", 1_000_000, 50.0, log2w=22),
        # genome estimate of an isolate's raw sample, once per isolate
        _case("estimate_5mbp", "estimate", 5_000_000, 9.5, k=21, gc=0.51, repeats=7),
        # unitigs of a finished table, once per k
        _case("compact_1mbp_50x_k31", "compact", 1_000_000, 50.0, log2w=22),
        # reads that still matter for the next k of the ladder
        _case("filter_1mbp_50x_k31", "filter", 1_000_000, 50.0, log2w=22),
        # a FASTQ pair into a device bank
        _case("ingest_1mbp_50x", "ingest", 1_000_000, 50.0),
        # a small cohort of uneven depth, two of them subsampled
        _case("batch_6", "batch", 300_000, 100.0, log2w=20, isolates=6),
    ]


def draw(rng):
    kind = rng.choice(["build"] * 6 + ["sketch", "estimate", "compact", "filter", "ingest", "batch"])
    lo, hi = {"build": (8e3, 5e6), "sketch": (5e4, 2e6), "estimate": (5e4, 6e6), "compact": (2e4, 1e6), "filter": (2e4, 1e6),
              "ingest": (1e4, 1e6), "batch": (5e4, 3e5)}[kind]
    genome = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    most = {"build": 100.0, "compact": 50.0, "filter": 50.0, "ingest": 50.0, "batch": 100.0, "sketch": 50.0, "estimate": 0.0}[kind]
    cov = 1.02 * 2 * READ_LEN * SAMPLE_PAIRS / genome if kind == "estimate" else math.exp(rng.uniform(math.log(20.0), math.log(most)))
    # the dynamic k ladder's values, the benchmark's, and odd ones between
    k = rng.choice([21, 25, 31, 33, 41, 55, 63, 65, 77, 91, 99, 127]) if kind in ("build", "sketch") else rng.choice([21, 31, 45])
    log2w = 0 if rng.random() < 0.5 else max(16, min(24, int(genome * 3).bit_length()))
    return dict(kind=kind, genome=genome, cov=round(cov, 2), k=31 if kind == "batch" else k, sub=rng.choice([0.001, 0.003, 0.005, 0.01]),
                gc=round(rng.uniform(0.3, 0.68), 2), cb=rng.choice([4, 16]) if kind != "batch" else 16,
                log2w=(log2w or 20) if kind == "batch" else log2w,
                tsc=rng.choice([0, 0, 0, 2, 5]) if kind == "build" else 0, repeats=rng.choice([0, 3, 7]),
                isolates=rng.randint(2, 6) if kind == "batch" else 1, hll_p=rng.choice([14, 16]) if kind == "estimate" else 14)


def _synth(case, seed, i=0):
    genome = case["genome"]
    kw = dict(seed=(seed * 1000003 + 7919 * i + 1) % (1 << 62), genome_len=genome, gc=case["gc"], coverage=case["cov"],
              sub_rate=case["sub"], indel_rate=0.0)
    if case["kind"] == "batch":  # uneven members: genome x 0.5 .. 1.5, depth x 0.3 .. 1.9
        r = np.random.default_rng([seed, i])
        kw.update(genome_len=int(genome * r.uniform(0.5, 1.5)), coverage=float(case["cov"] * r.uniform(0.3, 1.9)),
                  gc=float(r.uniform(0.30, 0.68)))
    if case["repeats"]:
        kw.update(n_repeats=case["repeats"], repeat_len=max(200, min(5000, genome // 50)), repeat_identity=0.99)
    return api.synth_params(**kw)


def _row_buffers(case):
    """Page-locked buffers with room for a table's rows, as a program that exports many tables keeps them."""
    g, k = case["genome"], case["k"]
    rows = int(g * (2.5 if case["kind"] == "batch" else 3.0 if 0 < case["tsc"] < 3 else 1.3)) + 65536
    nw = api.key_bits_for_k(k) // 64
    pin = lambda shape, dt: torch.empty(shape, dtype=dt, pin_memory=True).numpy()  # noqa: E731
    return pin((rows, nw), torch.int64).view(np.uint64), pin((rows,), torch.int16).view(np.uint16), pin((rows,), torch.uint8)


def _build(s, keep_cms=False):
    c = s["case"]
    return api.build_cdbg_ext(s["bank"], c["k"], c["tsc"] or None, c["genome"], ctx=context(), counter_bits=c["cb"],
                              cms_log2_width=c["log2w"], keep_cms=keep_cms)


def prepare(case, seed):
    ctx, kind = context(), case["kind"]
    s = dict(case=case)
    if kind == "ingest":
        d = tempfile.mkdtemp(prefix="fq_", dir="/dev/shm" if os.path.isdir("/dev/shm") else None)
        s["r1"], s["r2"] = os.path.join(d, "r1.fastq"), os.path.join(d, "r2.fastq")
        api.synth_write_fastq(_synth(case, seed), s["r1"], s["r2"])
        s["files"] = _Files(d, s["r1"], s["r2"])
        reads, words = int(case["genome"] * case["cov"] / READ_LEN) + 64, int(case["genome"] * case["cov"] / 32) + 64
        s["out"] = [np.zeros(words, np.uint64), np.zeros(reads, np.uint64), np.zeros(reads, np.uint32), np.zeros(reads, np.uint32)]
        return s
    if kind == "batch":
        s["members"] = [api.synth_isolate(_synth(case, seed, i), sample_pairs=SAMPLE_PAIRS) for i in range(case["isolates"])]
        s["rows"] = _row_buffers(case)
        return s
    bank, _, sample, n_sample, stats = api.synth_isolate(_synth(case, seed), sample_pairs=SAMPLE_PAIRS if kind == "estimate" else 0)
    if kind == "estimate":
        s.update(lengths=np.ascontiguousarray(sample.lengths), sample=sample, n_sample=n_sample, stats=stats,
                 bank=api.DeviceBank(ctx, sample))
        return s
    s["bank"] = api.DeviceBank(ctx, bank)
    if kind in ("build", "sketch"):
        s["rows"] = _row_buffers(case)
    else:
        s["table"] = _build(s)
        if kind == "filter":
            s["unitigs"], _, s["circular"], s["edges"] = api.compact(s["table"])
            s["table"].release()
            s["out"] = np.zeros(int(case["genome"] * case["cov"] / READ_LEN) + 64, np.uint8)
        else:
            s["out"] = [np.zeros(2 * case["genome"] + 65536, np.uint8), np.zeros(case["genome"] // 8 + 4096, np.uint8),
                        np.zeros((case["genome"] // 8 + 4096, 6), np.int64)]
    return s


class _Files:
    """The FASTQ pair on disk, gone with the state."""

    def __init__(self, d, *files):
        self.d, self.files = d, files

    def __del__(self):
        for f in self.files:
            if os.path.exists(f):
                os.unlink(f)
        if os.path.isdir(self.d):
            os.rmdir(self.d)


def _into(buf, x):
    """x at the start of a buffer whose size does not depend on the seed."""
    buf[:len(x)] = x
    buf[len(x):] = 0
    return buf


def _in_order(state, rows):
    """The exported rows on the device in an order of their own (a table has none): by a
    64-bit mix of the key's words; then zeros up to a size that does not depend on the seed."""
    keys, cov, mask = rows
    k = torch.from_numpy(keys.view(np.int64)).cuda(non_blocking=True)
    c = torch.from_numpy(cov.view(np.int16)).cuda(non_blocking=True)
    m = torch.from_numpy(mask).cuda(non_blocking=True)
    h = k[:, 0]
    for j in range(1, k.shape[1]):
        h = (h ^ (h >> 29)) * 0x1E3779B97F4A7C15 + k[:, j]
        h = (h ^ (h >> 32)) * 0x3F58476D1CE4E5B9
    o = torch.argsort(h)
    n, cap = len(o), len(state["rows"][1])
    out = k.new_zeros((cap, k.shape[1])), c.new_zeros(cap), m.new_zeros(cap)
    for x, y in zip(out, (k, c, m)):
        torch.index_select(y, 0, o, out=x[:n])
    return out


def _cycle(x):
    """A circular sequence from its smallest rotation on either strand (error cycles are short)."""
    rc = x[::-1].translate(bytes.maketrans(b"ACGT", b"TGCA"))
    return min(min(y[i:] + y[:i] for i in range(len(y))) for y in (x, rc))


def run(state):
    case, ctx = state["case"], context()
    kind = case["kind"]
    if kind == "build":
        t = _build(state)
        out = _in_order(state, t.export(out=state["rows"])), len(t), t.pushes()
        t.release()
        return out
    if kind == "sketch":
        t, cms = _build(state, keep_cms=True)
        out = _in_order(state, t.export(out=state["rows"])), cms.export(), t.info()[0]
        t.release()
        cms.release()
        return out
    if kind == "estimate":
        e, rt, rs = api.estimate_bank(ctx, state["bank"], state["lengths"], state["n_sample"], state["stats"], want_registers=True,
                                      max_pairs=MAX_PAIRS, target_cov=TARGET_COV, hll_p=case["hll_p"])
        return dict(genome_size=e.genome_size, u_ge_1=e.u_ge_1, u_ge_2=e.u_ge_2, pairs=e.pairs_sampled, m=e.m_sample, kmers=e.kmers,
                    cov=e.estimated_cov, factor=e.subsample_factor, depth=e.sample_kmer_depth, regs_total=rt, regs_solid=rs)
    if kind == "compact":
        # A unitig's coverage leaves out the last node of the walk, and which end the walk
        # starts from is not fixed (nor is it in the reference): it is not compared here.
        seqs, _, circular, edges = api.compact(state["table"])
        seqs = [_cycle(x) if c else x for x, c in zip(seqs, circular)]
        # unitigs in the order of their sequences, edges by those ranks
        o = sorted(range(len(seqs)), key=seqs.__getitem__)
        rank = np.empty(len(o) + 1, np.int64)
        rank[o] = np.arange(len(o))
        e = edges.astype(np.int64)
        e[:, 0], e[:, 2] = rank[e[:, 0]], rank[e[:, 2]]
        e = e[np.lexsort(e.T[::-1])]
        text = np.frombuffer(b"\n".join(seqs[i] for i in o), np.uint8)
        return len(o), len(e), [_into(b, x) for b, x in zip(state["out"], (text, circular[o], e))]
    if kind == "filter":
        keep, kept = api.filter_active_reads(ctx, state["bank"], state["unitigs"], state["circular"], state["edges"], case["k"])
        return _into(state["out"], keep), kept
    if kind == "ingest":
        bank, st, merged = api.ingest_fastq_device(ctx, state["r1"], state["r2"])
        *arrays, counts = bank.export()
        out = [_into(b, x) for b, x in zip(state["out"], arrays)], counts, merged, st.input_read_pairs, st.retained_read_pairs, st.merged_pairs_count, st.bases_after_trim
        bank.release()
        return out
    b = api.Batch(ctx, api.batch_params(policy=api.subsample_policy(**POLICY), k=case["k"], key_bits=api.key_bits_for_k(case["k"]),
                                        cms_log2_width=case["log2w"]))
    ids = [b.submit(bank, sample, n, stats) for bank, _, sample, n, stats in state["members"]]
    b.run()
    out = []
    for i in ids:
        t = b.take_table(i)
        out.append((_in_order(state, t.export(out=state["rows"])), b.result(i).subsample_factor))
        t.release()
    b.release()
    return out


def work(case):
    """Bytes of the packed reads (or FASTQ text) read once and of the results written once."""
    bases = case["genome"] * case["cov"]
    reads = bases / READ_LEN
    bank = bases / 4 + 16 * reads
    rows = case["genome"] * (api.key_bits_for_k(case["k"]) // 8 + 3)
    kind = case["kind"]
    if kind == "build":
        b = bank + rows
    elif kind == "sketch":
        b = bank + rows + (8 << (case["log2w"] or 20))
    elif kind == "estimate":
        b = min(bases, 2 * SAMPLE_PAIRS * READ_LEN) / 4 + (2 << case["hll_p"])
    elif kind == "compact":
        b = rows + 1.1 * case["genome"]
    elif kind == "filter":
        b = bank + reads + case["genome"]
    elif kind == "ingest":
        b = bases * 2.2 + bank
    else:
        b = case["isolates"] * (1.1 * bank + rows)
    return dict(bytes=float(b), flops=0.0)


# --- the estimator in 64 bits (estimator.rs:296-440), plain torch -----------------
_SEED = (0x3C8BFBB395C60474, 0x3193C18562A02B4C, 0x20323EE046061444, 0x295C504FAC61002E)
_ROWS = (0x243F6A8885A308D3, 0x13198A2E03707344, 0xA4093822299F31D0, 0x082EFA98EC4E6C89)


def _i64(x):
    x &= (1 << 64) - 1
    return x - (1 << 64) if x >> 63 else x


def _shr(x, n):
    return (x >> n) & ((1 << (64 - n)) - 1)


def _mix(z):
    z = (z ^ _shr(z, 30)) * _i64(0xBF58476D1CE4E5B9)
    z = (z ^ _shr(z, 27)) * _i64(0x94D049BB133111EB)
    return z ^ _shr(z, 31)


def _hll(regs):
    m = float(len(regs))
    raw = 0.7213 / (1.0 + 1.079 / m) * m * m / float(np.exp2(-regs.astype(np.float64)).sum())
    zeros = int((regs == 0).sum())
    return m * math.log(m / zeros) if raw <= 2.5 * m and zeros else raw


def exact(case, seed):
    """The estimate's floating values (everything else is whole numbers, which are compared as they are)."""
    if case["kind"] != "estimate":
        return None
    s = prepare(case, seed)
    k, p, n, lens, st = 21, case["hll_p"], s["n_sample"], s["lengths"].astype(np.int64), s["stats"]
    words = torch.from_numpy(s["sample"].data.view(np.int64)).cuda()
    codes = ((words[:, None] >> (2 * torch.arange(32, device="cuda"))) & 3).reshape(-1)
    nk = np.maximum(lens[:2 * n] - k + 1, 0)
    total = int(nk.sum())
    start = torch.from_numpy(s["sample"].offsets[:2 * n].astype(np.int64) - (np.cumsum(nk) - nk)).cuda()
    pos = torch.repeat_interleave(start, torch.from_numpy(nk).cuda()) + torch.arange(total, device="cuda")
    f, r = torch.zeros(total, dtype=torch.int64, device="cuda"), torch.zeros(total, dtype=torch.int64, device="cuda")
    rot = lambda v, q: _i64((v << (q % 64)) | (v >> ((64 - q) % 64))) if q % 64 else _i64(v)  # noqa: E731
    for j in range(k):
        c = codes[pos + j]
        f ^= torch.tensor([rot(v, k - 1 - j) for v in _SEED], device="cuda")[c]
        r ^= torch.tensor([rot(v, j) for v in _SEED[::-1]], device="cuda")[c]
    low = torch.tensor(_i64(1 << 63), device="cuda")
    raw = torch.where((f ^ low) < (r ^ low), f, r)
    t = torch.arange(total, device="cuda")
    solid = torch.ones(total, dtype=torch.bool, device="cuda")
    for seed_r in _ROWS:
        col = _mix(raw ^ _i64(seed_r)) & ((1 << 23) - 1)
        first = torch.full((1 << 23,), total, dtype=torch.int64, device="cuda").scatter_reduce_(0, col, t, "amin")
        solid &= first[col] < t
    h = _mix(raw)
    idx, rest = _shr(h, 64 - p), h & ((1 << (64 - p)) - 1)
    top = torch.floor(torch.log2((rest >> 20).double() + 0.5)).long() + 20  # the highest set bit, where it is above bit 20
    rho = torch.where(rest >> 20 > 0, 64 - p - top, 64 - p + 1)
    for b in range(21):
        rho = torch.where((rest >> 20 == 0) & (rest >> b > 0), 64 - p - b, rho)
    regs = [np.zeros(1 << p, np.int64), np.zeros(1 << p, np.int64)]
    pair_end = np.cumsum(nk)[1::2]
    use, done, a = min(n, MAX_PAIRS), 0, 0
    for stop in [*range(6000, use + 1, 2000), use]:
        e = int(pair_end[stop - 1])
        for w, sel in enumerate((slice(a, e), torch.nonzero(solid[a:e])[:, 0] + a)):
            x = torch.zeros(1 << p, dtype=torch.int64, device="cuda").scatter_reduce_(0, idx[sel], rho[sel], "amax")
            regs[w] = np.maximum(regs[w], x.cpu().numpy())
        a, done = e, stop
        u1, u2 = (round(_hll(x)) for x in regs)
        lam = max(0, e - max(0, u1 - u2)) / u2 if u2 else 0.0
        if lam >= 15.0 and stop % 2000 == 0 and stop >= 6000:
            break
    p2 = 1.0 - (1.0 + lam) * math.exp(-lam)
    g = max(10000, round(u2 / p2) if p2 > 0.05 else u2)
    cov = st.total_bases / g
    factor = min(max(TARGET_COV / cov, 0.01), 1.0) if cov > 1.5 * TARGET_COV else 1.0
    return dict(genome_size=None, u_ge_1=None, u_ge_2=None, pairs=None, m=None, kmers=None, cov=cov, factor=factor, depth=lam,
                regs_total=None, regs_solid=None)
