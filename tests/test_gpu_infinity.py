"""FP32: an infinity in the signal reaches the windows that hold it, not the
recomputed coefficients of the windows that end before it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# A run of 32 lags that an amplitude step makes recompute directly, at the end
# of the 8,192 samples whose statistics are taken together (254 runs of a
# shortest length of 64), with an infinity after its first windows of the
# longer template.  Lengths with a last piece of 1, 8 and 31 samples, and
# whole pieces.  Bound: that of the FP32 path.
@pytest.mark.parametrize("L", [993, 1000, 1023, 1024])
@pytest.mark.parametrize("value", [np.inf, -np.inf])
def test_windows_before_an_infinity(gpu, oracle, rng, L, value):
    n, lag0, clean = 20_000, 32 * 253, 6
    at = lag0 + clean - 1 + L  # the sample after the run's first `clean` windows
    x = rng.standard_normal(n) * np.where(np.arange(n) < lag0 + 4, 1.0, 1e-3)
    x = x.astype(np.float32)
    x[at] = value
    tps = [rng.standard_normal(64), rng.standard_normal(L)]
    p = gpu.SingleChannel.MatchedFilterParameters()
    for t in tps:
        w = gpu.WaveformTemplate()
        w.set_signal(t)
        w.set_sampling_rate(100.0)
        p.add_template(w)
    p.set_signal_size(n)
    f = gpu.SingleChannel.MatchedFilter(dtype=np.float32)
    f.initialize(p, correlator_variant=1)
    f.set_signal(x)
    f.apply()
    for t, tp in enumerate(tps):
        r = f.get_valid_matched_filtered_signal(t)[lag0:lag0 + 32].astype(np.float64)
        ref = oracle.pearson_naive(tp, x[lag0:lag0 + clean - 1 + tp.size])
        assert ref.size == clean
        assert np.max(np.abs(r[:clean] - ref)) < 1e-5, (t, r[:clean], ref)
    assert not np.any(np.abs(r[clean:]) > 0)


# batches whose longest template is shorter than a piece, just one piece, and one
# sample more: runs in the quiet part of a block are recomputed
@pytest.mark.parametrize("lens", [(5, 31), (31,) * 17, (32, 7), (33, 32, 31)])
def test_short_batches(gpu, oracle, rng, lens):
    n = 12_000
    x = (rng.standard_normal(n) * np.where(np.arange(n) < 5000, 1.0, 3e-4)).astype(np.float32)
    tps = [rng.standard_normal(L) for L in lens]
    p = gpu.SingleChannel.MatchedFilterParameters()
    for t in tps:
        w = gpu.WaveformTemplate()
        w.set_signal(t)
        w.set_sampling_rate(100.0)
        p.add_template(w)
    p.set_signal_size(n)
    f = gpu.SingleChannel.MatchedFilter(dtype=np.float32)
    f.initialize(p, correlator_variant=1)
    f.set_signal(x)
    f.apply()
    assert f.get_fixup_runs() > 0
    for t, tp in enumerate(tps):
        r = f.get_valid_matched_filtered_signal(t).astype(np.float64)
        lag = slice(5000, 5400)  # the quiet lags of a block with a loud part
        assert np.max(np.abs(r - oracle.pearson_naive(tp, x))[lag]) < 1e-5
