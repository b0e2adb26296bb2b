"""FP32 window normalisation: how much rounding its sums add up."""
import numpy as np
import pytest

from test_gpu_paths import _filter, _pearson

pytestmark = pytest.mark.gpu


# Templates of slow noise, whose windows have a mean of their own, copied into a
# quiet signal at 1,000 times their level, and the coefficients where the copies
# lie (all 1 but for the quiet signal): their error is that of the normalisation.
# In an FP32 emulation on the CPU (40 templates) the window sums err by 1.6e-7
# with the window's edges summed apart, 5.0e-7 and 5.3e-7 with the edge samples
# added one by one to the whole and with everything in sequence.  The transform
# spreads its rounding over the block, where the copies are few: below 0.5e-7 of
# a coefficient of 1, like the reciprocal square root and three products
# together.  The bound is twice the first figure.
def test_window_sums(gpu, rng):
    n, nch, L = 30_000, 48, 500
    x = 0.01 * rng.standard_normal((nch, n))
    tps, at = [], []
    for c in range(nch):
        tp = np.convolve(rng.standard_normal(L + 40), np.hanning(41), "valid")
        tps.append(tp / tp.std())
        at.append([])
        i = int(rng.integers(200, 1000))
        while i + L + 600 <= n:
            x[c, i:i + L] += tps[c]
            at[c].append(i)
            i += L + int(rng.integers(500, 1000))
    x = (x + 1e3).astype(np.float32)
    f = _filter(gpu, tps, list(range(nch)), nch, n, np.float32, correlator_variant=1)
    f.set_channel_signals(x)
    f.apply()
    rel = []
    for c in range(nch):
        ref, _ = _pearson(tps[c], x[c].astype(np.float64))
        rel.append(f.get_valid_matched_filtered_signal(c)[at[c]] / ref[at[c]] - 1.0)
    rms = float(np.sqrt(np.mean(np.concatenate(rel) ** 2)))
    print("relative error of the coefficients: %.3g" % rms)
    assert rms < 3.2e-7
