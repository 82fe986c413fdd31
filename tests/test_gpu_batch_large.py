"""A batch whose large isolates are built on their own, over minimizer bins, and whose small
ones share waves: every result field and row equals the single-isolate calls' and those of a
batch that takes all of them through the waves (integers, tolerance 0)."""
import pytest

from fastbact_gb300 import api
from test_gpu_batch import POLICY, check_same, run_batch, single

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
