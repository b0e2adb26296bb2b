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
