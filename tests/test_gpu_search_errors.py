"""A failed apply is reported by a peak search that has no lag to look at."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_empty_search_reports_a_failed_apply(gpu, rng, dtype):
    """The signal is shorter than the longest template: the common trace is
    empty, the shorter template has been correlated all the same."""
    from mflib_gb300 import _lib
    n = 300
    p = gpu.SingleChannel.MatchedFilterParameters()
    for L in (40, 400):
        w = gpu.WaveformTemplate()
        w.set_signal(rng.standard_normal(L))
        w.set_sampling_rate(100.0)
        p.add_template(w)
    p.set_signal_size(n)
    f = gpu.SingleChannel.MatchedFilter(dtype=dtype)
    f.initialize(p)
    f.set_signal(rng.standard_normal(n).astype(dtype))
    _lib.call("mfgpu_mf_test_wait_timeout", f._h)  # the correlator's copy is never issued: its bounded wait ends
    f.apply()
    with pytest.raises(_lib.MfgpuTimeout):
        f.find_peaks(0.5, 10)
    assert not f.have_matched_filtered_signals()
    f.apply()
    f.find_peaks(0.5, 10)
    assert f.get_peaks(0).size == 0 and f.get_peaks(1).size == 0
