"""DBSCAN of one feature with weights: the one-CTA form against the general
launches (taken by every segment of a call that holds one of more than 8,192
points), and its time in dense segments."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BIG = 8193


def _both(gpu, eps, mo, x, off, w):
    """Labels and cluster counts by the two forms."""
    db = gpu.DBSCAN()
    db.initialize(eps, mo)
    labels, ncl = db.cluster_segments(x, off, w)
    more = np.linspace(0.0, 1e9, BIG)
    xg, wg = np.concatenate([x, more]), None if w is None else np.concatenate([w, np.ones(BIG)])
    lg, ng = db.cluster_segments(xg, np.concatenate([off, [xg.size]]).astype(np.int32), wg)
    return (np.asarray(labels), np.asarray(ncl)), (np.asarray(lg)[:x.size], np.asarray(ng)[:-1])


# weights that are no binary fractions (a neighbourhood's sum depends on its
# order where it meets min_obs), equal ones, magnitudes far apart, infinities and
# values that are no numbers
@pytest.mark.parametrize("kind", ["tenths", "thirds", "wide", "special"])
@pytest.mark.parametrize("span", [0.02, 0.3, 3.0])
def test_forms_agree(gpu, rng, kind, span):
    sizes = (1, 2, 33, 1023, 1025, 8192)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    x = np.concatenate([np.round(rng.uniform(0, span * m, m) * 8) / 8 for m in sizes])
    w = {"tenths": lambda: rng.integers(1, 12, x.size) / 10.0,
         "thirds": lambda: np.full(x.size, 1.0 / 3.0),
         "wide": lambda: 10.0 ** rng.uniform(-12, 6, x.size),
         "special": lambda: np.where(rng.random(x.size) < 0.01, np.nan, np.where(rng.random(x.size) < 0.01, np.inf, 0.7))}[kind]()
    for eps, mo in ((0.25, 1), (1.0, 3), (5.0, 40)):
        (l1, n1), (l2, n2) = _both(gpu, eps, mo, x, off, w)
        np.testing.assert_array_equal(n1, n2)
        np.testing.assert_array_equal(l1, l2)


def test_a_dense_segment_takes_no_longer_with_weights(gpu, rng):
    """8,192 points in one neighbourhood: within five times the time without
    weights (the same number of neighbourhood sums, each from two loads)."""
    x, off = np.round(rng.uniform(0, 40.0, 8192)), np.array([0, 8192], np.int32)
    db = gpu.DBSCAN()
    db.initialize(50.0, 3)
    best = {}
    for name, w in (("none", None), ("weights", rng.uniform(0.5, 2.0, 8192))):
        best[name] = 1e9
        for _ in range(6):
            t = time.perf_counter()
            db.cluster_segments(x, off, w)
            best[name] = min(best[name], time.perf_counter() - t)
    assert best["weights"] < 5 * best["none"], best


def _lane_sums(values, places):
    """Sums as a warp forms them: the value at place j by lane j mod 32, then a tree over the lanes."""
    acc = np.zeros((len(values), 32))
    for k in range(values.shape[1]):
        acc[np.arange(len(values)), places[:, k] % 32] += values[:, k]
    for o in (16, 8, 4, 2, 1):
        acc = acc + acc[:, np.arange(32) ^ o]
    return acc[:, 0]


def test_weights_beside_a_nan_are_summed_in_the_points_order(gpu, rng):
    """Data holding a NaN are scanned in the points' own order.  Groups of
    points whose weights, sevenths, add up to min_obs but for rounding: each
    decides as that sum does."""
    groups, m, mo = 600, 12, 3
    k = rng.integers(1, 3, (groups, m))
    k[:, -1] = 7 * mo - k[:, :-1].sum(axis=1)
    k = k[k[:, -1] > 0]
    groups = len(k)
    place = np.sort(rng.permutation(groups * m).reshape(groups, m), axis=1) + 1  # the points of each group
    x, w = np.full(groups * m + 1, np.nan), np.ones(groups * m + 1)
    x[place] = 100.0 * np.arange(groups)[:, None]
    w[place] = k / 7.0
    values = w[place]
    core = _lane_sums(values, place) >= mo
    by_value = _lane_sums(values, m * np.arange(groups)[:, None] + np.arange(m)) >= mo
    assert np.any(core != by_value)
    db = gpu.DBSCAN()
    db.initialize(1.0, mo)
    labels, ncl = db.cluster_segments(x, np.array([0, x.size], np.int32), w)
    assert ncl[0] == core.sum()
    np.testing.assert_array_equal(np.asarray(labels)[place] >= 0, core[:, None].repeat(m, 1))


# more segments than the chip holds large CTAs: small CTAs, by the largest
# segment (their limits are 256 and 1,024 points), empty segments and segments
# of one point among them; few points beside one large segment
@pytest.mark.parametrize("largest,few", [(3, False), (256, False), (257, False), (1024, False), (1025, False), (1025, True)])
@pytest.mark.parametrize("weighted", [False, True])
def test_many_segments(gpu, rng, largest, few, weighted):
    sizes = rng.integers(0, 3 if few else min(largest, 40) + 1, 400)
    sizes[[7, 123, 399]] = largest, 0, 1
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    x = np.concatenate([np.round(rng.uniform(0, 0.5 * m, m) * 8) / 8 for m in sizes])
    x[::97], x[1::89], x[2::83] = np.nan, np.inf, -0.0
    w = rng.integers(1, 12, x.size) / 10.0 if weighted else None
    for eps, mo in ((0.25, 1), (1.0, 3)):
        (l1, n1), (l2, n2) = _both(gpu, eps, mo, x, off, w)
        np.testing.assert_array_equal(n1, n2)
        np.testing.assert_array_equal(l1, l2)


def test_many_small_segments_take_no_longer_than_the_general_form(gpu, rng):
    """100,000 segments of two points, in one call and beside a segment that
    sends them all to the general launches."""
    db = gpu.DBSCAN()
    db.initialize(50.0, 3)
    nseg = 100_000
    x, off = np.round(rng.uniform(0, 500, 2 * nseg)), (2 * np.arange(nseg + 1)).astype(np.int32)
    xg, og = np.concatenate([x, np.zeros(BIG)]), np.concatenate([off, [2 * nseg + BIG]]).astype(np.int32)
    best = {}
    for name, a, o in (("small", x, off), ("general", xg, og)):
        best[name] = 1e9
        for _ in range(6):
            t = time.perf_counter()
            db.cluster_segments(a, o, None)
            best[name] = min(best[name], time.perf_counter() - t)
    assert best["small"] < best["general"], best


# many points that are not core, with core neighbours of one or two clusters far
# from them in order
@pytest.mark.parametrize("weighted", [False, True])
def test_border_points(gpu, oracle, rng, weighted):
    n = 3000
    x = np.concatenate([rng.uniform(0, 4000, n - 40), rng.uniform(4600, 4700, 20), rng.uniform(5200, 5300, 20)]).round()
    x = x[rng.permutation(n)]
    w = rng.integers(1, 5, n) / 2.0 if weighted else None
    db = gpu.DBSCAN()
    for eps, share in ((1000.0, 0.45), (1000.0, 0.3), (700.0, 0.3), (50.0, 0.0245)):
        mo = int(share * n * (1.25 if weighted else 1.0))
        db.initialize(eps, mo)
        labels, ncl = db.cluster_segments(x, np.array([0, n], np.int32), w)
        n_ref, ref = oracle.dbscan(x, eps, mo, w)
        assert ncl[0] == n_ref
        np.testing.assert_array_equal(np.asarray(labels), ref)
    assert n_ref > 1
