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


# window variances in runs of 32 lags: every remainder of the length modulo 4,
# the shortest and longest of one and two runs per thread, a constant stretch
# inside the data (its windows give exactly 0) next to windows that leave it.
# Bound: the flagging bound's, as above.
@pytest.mark.parametrize("L", [64, 65, 66, 67, 93, 95, 96, 128, 500, 501, 4062, 4063, 4064, 4065, 4099])
def test_window_variances(gpu, oracle, rng, L):
    n = 30_011
    x = (rng.standard_normal(n) + 20.0).astype(np.float32)
    x[9_000:9_000 + L + 777] = 3.0
    tp = rng.standard_normal(L)
    f = _filter(gpu, [tp], [0], 1, n, np.float32, correlator_variant=1)
    f.set_channel_signals(x[None, :])
    f.apply()
    r = f.get_valid_matched_filtered_signal(0)
    assert np.all(r[9_000:9_778] == 0.0)
    live = np.ones(n - L + 1, bool)
    live[9_000:9_778] = False
    ref = oracle.pearson_naive(tp, x)
    assert float(np.max(np.abs(r.astype(np.float64) - ref)[live])) < FP32_TOL


# work groups: channels with one template, uneven counts, more CTAs than one
# wave holds with the last channels split finer.  Every template's row is
# compared (a template in no group, or in two of one channel, shows).
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("per,n", [((1,), 3000), ((1, 0, 5, 33), 3000), ((31,) * 12 + (32,) * 4, 42_000), ((7, 64, 3), 90_000)])
@pytest.mark.parametrize("equal", [False, True])
def test_work_groups(gpu, oracle, rng, dtype, per, n, equal):
    x = rng.standard_normal((len(per), n)).astype(dtype)
    chan = [c for c, m in enumerate(per) for _ in range(m)]
    lens = [300 if equal else 200 + 13 * (t % 31) for t in range(len(chan))]
    tps = [rng.standard_normal(L) for L in lens]
    f = _filter(gpu, tps, chan, len(per), n, dtype)
    f.set_channel_signals(x)
    f.apply()
    for t in range(0, len(tps), 1 if n < 10_000 else 7):
        r = f.get_valid_matched_filtered_signal(t).astype(np.float64)
        assert float(np.max(np.abs(r - oracle.pearson_naive(tps[t], x[chan[t]])))) < (FP32_TOL if dtype == np.float32 else 1e-12)
    for t in range(len(tps)):  # rows written to the end
        assert np.any(f.get_valid_matched_filtered_signal(t)[-32:] != 0)


# FP64 banks of several lengths: integers, or buckets of FP64 transforms where
# one template would leave the others few lags per block.
@pytest.mark.parametrize("lens,integer", [((200,) * 20 + (4000,), False), ((200, 400, 3000) * 5, True), ((4065, 60), True)])
def test_integer_or_buckets(gpu, oracle, rng, lens, integer):
    n = 30_000
    x = rng.standard_normal((1, n))
    tps = [rng.standard_normal(L) for L in lens]
    f = _filter(gpu, tps, [0] * len(lens), 1, n, np.float64)
    f.set_channel_signals(x)
    f.apply()
    assert (f.get_plan()["correlator"] == 7) == integer
    assert _worst(f, oracle, tps, [x[0]] * len(lens)) < 1e-12


# tensor-core form: groups whose templates the four epilogue warpgroups share
# unevenly or not at all, partly filled groups, a tile of one lag, a dead
# channel.  Bound: the flagging bound's, as above.
@pytest.mark.parametrize("group,per", [(2, 1), (2, 3), (4, 3), (6, 6), (10, 9), (16, 15), (16, 18)])
def test_tensor_epilogue(gpu, oracle, rng, group, per):
    L, nch = 96, 3
    n = 5 * 1024 + L  # lags 0 .. 5 * 1024
    x = (rng.standard_normal((nch, n)) + 5.0).astype(np.float32)
    x[1] = 2.0
    tps = [rng.standard_normal(L) for _ in range(nch * per)]
    chan = [t % nch for t in range(nch * per)]
    for t in (0, nch * per - 1):  # coefficients near 1 and -1
        x[chan[t], 2000 + 7 * t:2000 + 7 * t + L] = (1 - 2 * (t & 1)) * 40.0 * tps[t] + 5.0
    f = _filter(gpu, tps, chan, nch, n, np.float32, correlator_variant=4, tc_group=group)
    f.set_channel_signals(x)
    f.apply()
    for t in range(nch * per):
        r = f.get_valid_matched_filtered_signal(t)
        if chan[t] == 1:
            assert np.all(r == 0.0)
        else:
            assert float(np.max(np.abs(r.astype(np.float64) - oracle.pearson_naive(tps[t], x[chan[t]])))) < FP32_TOL


# shift and stack in batches of eight rows: remainders of a batch, shifts
# before the first lag.  Sums of at most nt coefficients of magnitude 1 in the
# data type, weights that sum to 1: nt roundings.
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("nt", [1, 7, 8, 9, 17])
def test_stack_batches(gpu, oracle, rng, dtype, nt):
    n, L = 5003, 64
    x = rng.standard_normal((nt, n)).astype(dtype)
    p = gpu.MultiChannel.MatchedFilterParameters()
    shifts = [7 * t for t in range(nt)]
    for t in range(nt):
        w = gpu.WaveformTemplate()
        w.set_signal(rng.standard_normal(L))
        w.set_sampling_rate(100.0)
        w.set_phase_travel_time(1.0 + shifts[t] / 100.0)
        w.set_phase_onset_time_in_signal(1.0 if t else 0.0)
        p.add_template(w)
    shifts[0] += 100
    p.set_signal_size(n)
    f = gpu.MultiChannel.MatchedFilter(dtype=dtype)
    f.initialize(p)
    f.set_channel_signals(x)
    f.apply()
    rows = [f.get_matched_filtered_signal(t).astype(np.float64) for t in range(nt)]
    ref = oracle.shift_and_stack(rows, rows[0].size, shifts, [1] * nt)
    out = f.shift_and_stack()
    assert out.size == ref.size
    assert float(np.max(np.abs(out.astype(np.float64) - ref))) <= (nt + 2) * np.finfo(dtype).eps


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


def _pearson(tp, z):
    """Two-pass Pearson coefficients and window 2-norms about the mean, each
    window taken relative to its first sample (so that a small deviation on a
    large level keeps its digits)."""
    b = tp - tp.mean()
    b /= np.linalg.norm(b)
    w = np.lib.stride_tricks.sliding_window_view(z, tp.size)
    rho, norm = np.empty(w.shape[0]), np.empty(w.shape[0])
    for i in range(0, w.shape[0], 2048):
        d = w[i:i + 2048] - w[i:i + 2048, :1]
        d -= d.mean(axis=1, keepdims=True)
        norm[i:i + 2048] = np.sqrt((d * d).sum(axis=1))
        rho[i:i + 2048] = (d @ b) / norm[i:i + 2048]
    return rho, norm


# FP64 in integer arithmetic: the longest and shortest templates, block and
# tile edges (a last block of one lag), several lengths and one, offsets and
# scales near the ends of the FP64 range.  Bound: that of the reference's own
# tests (1e-13; the two-pass sums it is compared with err by about L 2^-53)
# plus, against the window's own deviation, the samples' rounding (at most
# 2^-50 of the signal's largest deviation each) and the rounding of the
# template's mean (its demeaned samples sum to up to L 2^-52 of it, times the
# window's level).
@pytest.mark.parametrize("lens,n", [((2,), 4097), ((500,), 3585 + 499), ((500,) * 3, 3584 + 499), ((31, 32, 33, 200), 9000),
                                    ((4065,), 4065), ((4065, 4064, 64), 8193 + 32), ((1000,) * 21, 16_385),
                                    ((2801, 700, 1500, 700), 20_000)])
@pytest.mark.parametrize("scale,offset", [(1.0, 0.0), (3e-2, 4e4), (1e-150, 0.0), (1e150, -1e150)])
def test_integer_correlator(gpu, oracle, rng, lens, n, scale, offset):
    x = rng.standard_normal((2, n))
    x[1] *= np.where(np.arange(n) < n // 2, 1.0, 40.0)
    tps = [rng.standard_normal(L) for L in lens]
    chan = [t % 2 for t in range(len(lens))]
    f = _filter(gpu, tps, chan, 2, n, np.float64)
    assert f.get_plan()["correlator"] == 7
    f.set_channel_signals(x * scale + offset)
    f.apply()
    if scale < 1e-100:
        # deviations below the normalisation's floor of 1e-12: coefficients
        # are the numerators over it
        assert all(np.max(np.abs(f.get_valid_matched_filtered_signal(t))) < 1e-130 for t in range(len(tps)))
        return
    # the coefficients do not depend on scale and offset; the reference is
    # taken on the samples as rounded, moved back to the middle of the range
    y = (x * scale + offset - offset) / scale if abs(scale) < 1e100 else x * scale / 1e150 + offset / 1e150
    tol = 1e-13 if abs(offset) <= scale * 1e3 else 1e-9  # digits the samples lost to the offset
    for t, tp in enumerate(tps):
        z = y[chan[t]]
        ref, norm = _pearson(tp, z)
        off = tp.size * 2.0 ** -52 * abs(tp.mean()) / np.linalg.norm(tp - tp.mean())
        bound = tol + (np.sqrt(tp.size) * 2.0 ** -50 + off) * np.max(np.abs(z - z.mean())) / norm
        err = np.abs(f.get_valid_matched_filtered_signal(t) - ref)
        assert np.all(err < bound), float(np.max(err / bound))


def test_integer_correlator_special_values(gpu, oracle, rng):
    n, L = 30_000, 300
    x = rng.standard_normal((3, n))
    x[0, 10_000] = np.nan
    x[1, 20_000] = -np.inf
    x[2, 9_000:15_000] = 7.25  # constant windows: 0
    tp = rng.standard_normal(L)
    f = _filter(gpu, [tp] * 3, [0, 1, 2], 3, n, np.float64)
    f.set_channel_signals(x)
    f.apply()
    S = f.get_plan()["lags_per_block"]
    for c, at in ((0, 10_000), (1, 20_000)):
        r = f.get_valid_matched_filtered_signal(c)
        assert np.all(np.isnan(r[at - L + 1:at + 1]))  # every window that holds it
        clean = np.where(np.isfinite(x[c]), x[c], 0.0)
        ref = oracle.pearson_naive(tp, clean)
        b = np.arange(r.size) // S * S
        far = (at < b) | (at >= b + 4096)  # blocks that do not read it
        assert np.max(np.abs(r[far] - ref[far])) < 1e-13
    r = f.get_valid_matched_filtered_signal(2)
    assert np.all(r[9_000:15_000 - L + 1] == 0.0)
    ref = oracle.pearson_naive(tp, x[2])
    keep = np.ones(r.size, bool)
    keep[9_000:15_000 - L + 1] = False
    assert np.max(np.abs(r[keep] - ref[keep])) < 1e-13


# association segments in one CTA each: sizes around the powers of two of the
# sorting network, up to the largest one CTA takes and one above it (the
# general launches), empty segments, ties, NaN, infinities, both zeros
@pytest.mark.parametrize("sizes", [(1, 2, 3, 0, 4, 5), (31, 32, 33, 1023, 1024, 1025), (8192, 8191, 7), (8193, 20)])
@pytest.mark.parametrize("weighted", [False, True])
def test_segment_clustering(gpu, oracle, rng, sizes, weighted):
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    x = np.round(rng.uniform(-off[-1] / 8, off[-1] / 8, off[-1]) * 4) / 4
    x[::37] = -0.0
    x[1::53] = np.inf
    x[2::59] = -np.inf
    if max(sizes) <= 8192:
        x[3::61] = np.nan
    w = rng.integers(1, 7, x.size) / 2.0 if weighted else None
    db = gpu.DBSCAN()
    for eps, mo in ((0.0, 1), (0.25, 3), (0.75, 6)):
        db.initialize(eps, mo)
        labels, ncl = db.cluster_segments(x, off, w)
        for s in range(len(sizes)):
            a, b = off[s], off[s + 1]
            if a == b:
                assert ncl[s] == 0
                continue
            n_ref, ref = oracle.dbscan(x[a:b], eps, mo, None if w is None else w[a:b])
            assert ncl[s] == n_ref
            np.testing.assert_array_equal(labels[a:b], ref)
