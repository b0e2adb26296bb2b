"""The two forms of the peak search (one CTA per trace, and rounds over all
traces for traces with more candidates than one CTA takes): which one runs, by
the launches that a search takes, and its peaks against the CPU oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THR = 0.125
FEW = 4  # launches of the one-CTA form: scan, totals, prune, emit


def _filter(mf, templates, n, dtype):
    p = mf.MultiChannel.MatchedFilterParameters()
    for t in templates:
        w = mf.WaveformTemplate()
        w.set_signal(t)
        w.set_sampling_rate(100.0)
        p.add_template(w)
    p.set_signal_size(n)
    f = mf.MultiChannel.MatchedFilter(dtype=dtype)
    f.initialize(p, template_channels=[0] * len(templates), n_channels=1)
    return f


def _search(f, oracle, thr, dist, templates):
    """Launches of a search, its peaks compared."""
    before = f.launch_count()
    f.find_peaks(thr, dist)
    used = f.launch_count() - before
    for t in templates:
        np.testing.assert_array_equal(f.get_peaks(t), oracle.peaks(f.get_matched_filtered_signal(t).astype(np.float64), thr, dist))
    return used


# one window of noise (hundreds of candidates in a chunk) between quiet ones:
# once a search has met few candidates again, the next one takes the short form
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("fused", [False, True])
def test_search_after_a_dense_one(gpu, oracle, rng, dtype, fused):
    n, L = 40_000, 200
    tps = [rng.standard_normal(L) for _ in range(3)]
    noise = rng.standard_normal((1, n)).astype(dtype)
    quiet = np.zeros((1, n), dtype)
    for i, t in enumerate(tps):
        quiet[0, 5000 + 9000 * i:5000 + 9000 * i + L] = t
    f = _filter(gpu, tps, n, dtype)
    if fused:
        f.set_peak_threshold(THR)
    used = []
    for x in (quiet, noise, noise, quiet, quiet, noise, quiet, quiet):
        f.set_channel_signals(x)
        f.apply()
        used.append(_search(f, oracle, THR, 50, range(3)))
    assert used[0] <= FEW and used[1] > FEW and used[2] > FEW and used[4] <= FEW and used[7] <= FEW, used


# more candidates in all traces together than the packed arrays hold at first
# (65,536), few in each: the arrays grow and the form stays
def test_many_traces_with_few_candidates_each(gpu, oracle, rng):
    nt, L, step = 300, 100, 400
    tp = rng.standard_normal(L)
    tps = [tp + 0.05 * rng.standard_normal(L) for _ in range(nt)]
    n = 250 * step
    x = 0.01 * rng.standard_normal(n)
    for i in range(0, n - L, step):
        x[i:i + L] += tp
    f = _filter(gpu, tps, n, np.float32)
    f.set_channel_signals(x[None, :].astype(np.float32))
    f.apply()
    first = _search(f, oracle, 0.875, 50, (0, nt - 1))
    assert int(np.sum(f.get_all_peaks()[0])) > 65_536
    assert first <= FEW + 2 and _search(f, oracle, 0.875, 50, (7, 150)) <= FEW
