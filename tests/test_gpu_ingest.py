"""The device ingest where its warp-wide forms can go wrong, against the oracle's restatement
(bytes and whole numbers, tolerance 0): reads at the edges of the words of its bit planes and
of the length up to which it uses them, overlaps of every length between none and all, equal
scores (repeats), adapters at every place, short and long ends of bad quality, and pair counts
at the edges of its tiles; texts with '\\r' and without a last newline, from memory and from
files."""
import ctypes as C
import os

import numpy as np
import pytest

from fastbact_gb300 import _native as N
from fastbact_gb300 import api
from test_gpu_parity import _check_device_ingest

pytestmark = pytest.mark.gpu
COMP = bytes.maketrans(b"ACGTacgtN", b"TGCAtgcaN")
LENS = [1, 9, 10, 14, 15, 16, 31, 32, 33, 63, 64, 65, 99, 100, 101, 109, 110, 111, 150, 511, 512, 513, 700]
ADAPTERS = [b"AGATCGGAAGAGC", b"AGATGTGTATAAGAGACAG", b"CTGTCTCTTATACACATCT"]


def rc(s):
    return s[::-1].translate(COMP)


def pairs(seed, n):
    rng = np.random.default_rng(seed)
    acgt = np.frombuffer(b"ACGT", np.uint8)
    out = []
    for i in range(n):
        l1 = int(rng.choice(LENS))
        l2 = l1 if rng.random() < 0.6 else int(rng.choice(LENS))
        frag = acgt[rng.integers(0, 4, int(rng.integers(max(l1, l2), l1 + l2 + 20)))].tobytes()
        if rng.random() < 0.2:  # repeats: several overlaps with the same score
            unit = frag[: int(rng.integers(1, 12))]
            frag = (unit * (len(frag) // len(unit) + 1))[: len(frag)]
        ends = []
        for r, L in ((frag, l1), (rc(frag), l2)):
            s = bytearray(r[:L])
            for j in np.flatnonzero(rng.random(len(s)) < rng.choice([0.0, 0.01, 0.08])):
                s[j] = int(rng.choice(np.frombuffer(b"ACGTNacgt", np.uint8)))
            if rng.random() < 0.3:
                ad = bytearray(ADAPTERS[int(rng.integers(3))])
                ad[int(rng.integers(10))] = int(rng.choice(acgt))
                j = int(rng.integers(0, len(s)))
                s[j:j + len(ad)] = ad[: len(s) - j]
            q = rng.integers(33 + 25, 33 + 41, len(s))
            tail = int(rng.integers(0, len(s) + 1)) if rng.random() < 0.4 else 0
            q[len(s) - tail:] = rng.integers(30, 33 + 22, tail)
            ends.append((bytes(s), q.astype(np.uint8).tobytes()))
        out.append(ends)
    return out


def text(ps, mate, eol=b"\n", last=True):
    t = b"".join(b"@p%d/%d" % (i, mate + 1) + eol + p[mate][0] + eol + b"+" + eol + p[mate][1] + eol for i, p in enumerate(ps))
    return t if last else t[: -len(eol)]


@pytest.mark.parametrize("n,opts", [(1, {}), (63, dict(min_len=1)), (64, dict(min_len=5, min_qual=0)), (65, dict(min_len=1, enable_merge=False)),
                                    (129, dict(min_len=1, enable_trim=False)), (700, dict(min_len=10)),
                                    (2000, dict(min_len=3, min_qual=15, subsample_factor=0.7, seed=5))])
def test_pairs_match_oracle(ctx, tmp_path, n, opts):
    kw = dict(subsample_factor=1.0, min_len=30, min_qual=20, enable_trim=True, enable_merge=True, seed=0)
    kw.update(opts)
    ps = pairs(1000 + n, n)
    if n == 1:
        ps = [[(b"ACGTTGCA" * 12, b"I" * 96), (rc(b"ACGTTGCA" * 12), b"I" * 96)]]
    r1, r2 = tmp_path / "e_1.fq", tmp_path / "e_2.fq"
    r1.write_bytes(text(ps, 0, last=n % 2 == 0))
    r2.write_bytes(text(ps, 1))
    bank, _ = _check_device_ingest(ctx, r1, r2, kw)
    # the same reads with '\r', from memory
    a, b = (np.frombuffer(text(ps, m, b"\r\n"), np.uint8) for m in (0, 1))
    h, st = C.c_void_p(), N.IngestStatsC()
    N.check(N.lib().fbk_ingest_fastq_device(ctx.handle, N.ptr(a), a.size, N.ptr(b), b.size, kw["subsample_factor"], kw["min_len"],
                                            kw["min_qual"], int(kw["enable_trim"]), int(kw["enable_merge"]), kw["seed"], C.byref(h),
                                            C.byref(st)), ctx.handle, "device ingest")
    crlf = api.DeviceBank.from_handle(ctx, h)
    for x, y in zip(bank.export(), crlf.export()):
        assert np.array_equal(x, y)
    bank.release()
    crlf.release()


@pytest.mark.parametrize("n", [40, 30_000])  # below and above the size that goes through the staging slots
def test_files_that_cannot_be_read(ctx, tmp_path, n):
    """A pipe, a closed or write-only descriptor and a directory in either place are refused;
    the same files are read afterwards, their positions unmoved."""
    ps = pairs(7, 40) * (n // 40)
    paths = [tmp_path / "e_1.fq", tmp_path / "e_2.fq"]
    for m, p in enumerate(paths):
        p.write_bytes(text(ps, m))
    assert (paths[0].stat().st_size > 4 << 20) == (n > 40)

    def ingest(fd1, fd2):
        h, st = C.c_void_p(), N.IngestStatsC()
        N.check(N.lib().fbk_ingest_fastq_fd_device(ctx.handle, fd1, fd2, 1.0, 1, 20, 1, 1, 0, C.byref(h), C.byref(st)), ctx.handle)
        return api.DeviceBank.from_handle(ctx, h), st

    r, w = os.pipe()
    write_only, folder = os.open(paths[1], os.O_WRONLY), os.open(tmp_path, os.O_RDONLY)
    good = [os.open(p, os.O_RDONLY) for p in paths]
    os.lseek(good[0], 17, os.SEEK_SET)
    closed = os.dup(r)
    os.close(closed)
    try:
        for bad in (r, closed, write_only, folder):
            for fds in ((bad, good[1]), (good[0], bad)):
                with pytest.raises(N.FbkError, match="FBK_ERR_IO"):
                    ingest(*fds)
        bank, st = ingest(*good)
        assert st.input_read_pairs == len(ps) and os.lseek(good[0], 0, os.SEEK_CUR) == 17
        a, b = (np.frombuffer(p.read_bytes(), np.uint8) for p in paths)
        h, st = C.c_void_p(), N.IngestStatsC()
        N.check(N.lib().fbk_ingest_fastq_device(ctx.handle, N.ptr(a), a.size, N.ptr(b), b.size, 1.0, 1, 20, 1, 1, 0, C.byref(h), C.byref(st)),
                ctx.handle)
        memory = api.DeviceBank.from_handle(ctx, h)
        for x, y in zip(bank.export(), memory.export()):
            assert np.array_equal(x, y)
        bank.release()
        memory.release()
    finally:
        for fd in (r, w, write_only, folder, *good):
            os.close(fd)
