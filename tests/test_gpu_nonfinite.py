"""Infinities and NaN in templates and signals."""
import numpy as np
import pytest

from test_gpu_paths import _filter, _pearson

pytestmark = pytest.mark.gpu


# a template that holds one has no coefficients; the bank's other templates keep
# theirs (bounds of the reference's own tests and of the FP32 path)
@pytest.mark.parametrize("dtype,tol", [(np.float64, 1e-12), (np.float32, 1e-5)])
@pytest.mark.parametrize("lens", [(300,) * 4, (300, 200, 411, 64)])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1.7e308])
def test_templates(gpu, rng, dtype, tol, lens, value):
    n = 6000
    x = rng.standard_normal((1, n)).astype(dtype)
    tps = [rng.standard_normal(L) for L in lens]
    tps[1][17] = value
    tps[2][:] = value
    f = _filter(gpu, tps, [0] * 4, 1, n, dtype)
    f.set_channel_signals(x)
    f.apply()
    for t in (0, 3):
        ref, _ = _pearson(tps[t], x[0].astype(np.float64))
        assert np.max(np.abs(f.get_valid_matched_filtered_signal(t) - ref)) < tol
    for t in (1, 2):
        r = f.get_valid_matched_filtered_signal(t)
        if not np.isfinite(value):
            assert np.all(np.isnan(r))
        else:  # samples whose mean or squares overflow: no coefficient stands out
            assert not np.any(np.abs(r) > 1e-6)


# FP64: the windows that hold one have no coefficient, the others are as accurate
# as without it, in its block too and where the whole signal is one block (in the
# reference signal it is a zero, 3 from the level; the samples' rounding as in
# the tests of the integer correlator).
@pytest.mark.parametrize("lens", [(2,), (33,), (300, 300), (300, 64, 150), (1500, 200)])
@pytest.mark.parametrize("n,at", [(1700, (0,)), (1700, (640, 641, 1699)), (14_000, (4095, 4096, 9000))])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_signals(gpu, rng, lens, n, at, value):
    x = rng.standard_normal(n) + 3.0
    tps = [rng.standard_normal(L) for L in lens]
    x[list(at)] = value
    f = _filter(gpu, tps, [0] * len(lens), 1, n, np.float64)
    assert f.get_plan()["correlator"] == 7
    f.set_channel_signals(x[None, :])
    f.set_peak_threshold(0.5)
    f.apply()
    clean = np.where(np.isfinite(x), x, 0.0)
    for t, tp in enumerate(tps):
        ref, norm = _pearson(tp, clean)
        r = f.get_valid_matched_filtered_signal(t)
        lag = np.arange(r.size)
        holds = np.zeros(r.size, bool)
        for i in at:
            holds |= (lag <= i) & (i < lag + tp.size)
        assert np.all(np.isnan(r[holds]))
        bound = 1e-13 + np.sqrt(tp.size) * 2.0 ** -50 * 10.0 / np.maximum(norm, 1e-300)
        assert np.all(np.abs(r - ref)[~holds] < bound[~holds])
