"""FP64 in integer arithmetic: how far a loud sample reaches."""
import numpy as np
import pytest

from test_gpu_paths import _filter, _pearson

pytestmark = pytest.mark.gpu


# One loud sample.  Blocks that do not read it are as accurate as without it
# (the bound of the reference's own tests); in a block that does, the samples'
# unit is 2^-54 of the loudest window at least (2^-55.1 and a power of two, with
# the estimate of the window norms above them), each sample is off by half a
# unit, a window by sqrt(L) of that, in the numerator and in the normalisation.
@pytest.mark.parametrize("lens", [(33,), (1500,), (2801,), (200, 1500), (2000, 64, 700, 2000)])
@pytest.mark.parametrize("loud", [1e3, 1e6, 1e9])
def test_a_loud_sample_and_the_blocks_around_it(gpu, rng, lens, loud):
    n = 24_000
    x = rng.standard_normal((1, n))
    tps = [rng.standard_normal(L) for L in lens]
    f = _filter(gpu, tps, [0] * len(lens), 1, n, np.float64)
    assert f.get_plan()["correlator"] == 7
    S = f.get_plan()["lags_per_block"]
    at = (4096 // S + 2) * S + 4096 + 20  # just past the end of a block
    x[0, at] += loud
    f.set_channel_signals(x)
    f.apply()
    for t, tp in enumerate(tps):
        ref, norm = _pearson(tp, x[0])
        err = np.abs(f.get_valid_matched_filtered_signal(t) - ref)
        first = np.arange(ref.size) // S * S
        reads = (at >= first) & (at < first + 4096)
        assert np.any(reads) and np.any(~reads & (first + 8192 > at) & (first < at))
        assert np.max(err[~reads]) < 1e-13, np.max(err[~reads])
        bound = 1e-13 + np.sqrt(tp.size) * 2.0 ** -53 * loud / norm
        assert np.all(err[reads] < bound[reads]), np.max(err[reads] / bound[reads])
