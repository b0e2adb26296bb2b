"""Kernels and dispatch branches at the sizes where they can go wrong (edges
of pieces and tiles, remainders, the smallest and largest of their ranges),
against the CPU oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FP32_TOL = 1e-5


def _filter(mf, templates, chan, nch, n, dtype, **kw):
    p = mf.MultiChannel.MatchedFilterParameters()
    for t in templates:
        w = mf.WaveformTemplate()
        w.set_signal(t)
        w.set_sampling_rate(100.0)
        p.add_template(w)
    p.set_signal_size(n)
    f = mf.MultiChannel.MatchedFilter(dtype=dtype)
    f.initialize(p, template_channels=chan, n_channels=nch, **kw)
    return f


def _worst(f, oracle, templates, sigs):
    """Largest deviation from the two-pass Pearson coefficient (the running
    sums of the reference's normalisation lose digits at amplitude steps)."""
    return max(float(np.max(np.abs(f.get_valid_matched_filtered_signal(t).astype(np.float64)
                                   - oracle.pearson_naive(templates[t], sigs[t]))))
               for t in range(len(templates)))


# listed runs: lengths around the 32-sample pieces, more templates than one
# batch holds, one piece up to the longest template an FFT plan takes.  The
# listed runs' own error is that of an FP32 dot product over the window
# (below 2^-24 sqrt(L) for unit-norm templates), the others are within the
# flagging bound of 2e-5 with its constant of 8 against 1.3 measured.
@pytest.mark.parametrize("lens", [(33,), (64,) * 17, (5, 31, 32, 33, 63, 64, 65, 96, 97, 200, 201, 223, 224, 225, 256,
                                                      999, 1000, 1001), (1000,) * 40, (3000, 8161)])
def test_listed_runs(gpu, oracle, rng, lens):
    n = 30_000
    x = (rng.standard_normal(n) * np.where(np.arange(n) < 14_321, 1.0, 3e-4) + 50.0).astype(np.float32)
    tps = [rng.standard_normal(L) for L in lens]
    f = _filter(gpu, tps, [0] * len(lens), 1, n, np.float32, correlator_variant=1)
    f.set_channel_signals(x[None, :])
    f.apply()
    assert f.get_fixup_runs() > 0
    assert _worst(f, oracle, tps, [x] * len(lens)) < FP32_TOL


# pruning per trace: traces without a candidate, with more than one CTA
# prunes (the general rounds take over) and with more candidates in a chunk
# than its slot holds; separations from none to the trace's length.  Indices
# are compared exactly, on the coefficients the search ran on.
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("thr,dist", [(0.0625, 0), (0.0625, 1), (0.03125, 7), (0.3125, 40), (0.3125, 50_000), (0.984375, 3)])
@pytest.mark.parametrize("fused", [False, True])
def test_prune_per_trace(gpu, oracle, rng, dtype, thr, dist, fused):
    n, lens = 41_007, (60, 300, 200, 300, 60)
    x = rng.standard_normal((2, n))
    x[1, 1000:9000] = 0.0
    tps = [x[t % 2, 20_000 + 500 * t:20_000 + 500 * t + L].copy() for t, L in enumerate(lens)]
    f = _filter(gpu, tps, [t % 2 for t in range(len(lens))], 2, n, dtype)
    f.set_channel_signals(x.astype(dtype))
    if fused:
        f.set_peak_threshold(thr)
    f.apply()
    for _ in range(2):
        f.find_peaks(thr, dist)
        for t in range(len(lens)):
            ref = oracle.peaks(f.get_matched_filtered_signal(t).astype(np.float64), thr, dist)
            np.testing.assert_array_equal(f.get_peaks(t), ref)
