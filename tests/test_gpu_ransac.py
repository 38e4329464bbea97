"""Batched RANSAC scoring on the GPU (uslam_ransac_score) against the
oracle: inlier counts and bitmasks of many fundamental matrices over the
correspondences of a synthetic two view geometry and of a real matched frame
pair, including ragged and empty match counts."""
import numpy as np
import pytest

import oracle
from uni_slam_gb300 import Context, synth

from test_oracle_ransac import two_view

pytestmark = pytest.mark.gpu


def _hypotheses(rs, p, q, h):
    """Fundamental matrices fitted (numpy 8-point, unnormalised) to random 8-samples."""
    out = []
    for _ in range(h):
        s = rs.choice(len(p), 8, replace=False)
        A = np.c_[q[s, 0:1] * p[s], q[s, 0:1], q[s, 1:2] * p[s], q[s, 1:2], p[s], np.ones((8, 1))]
        out.append(np.linalg.svd(A)[2][-1].reshape(3, 3))
    return np.array(out)


def test_ransac_score_equals_oracle(brief_pattern):
    rs = np.random.RandomState(9)
    F, p, q = two_view(rs, n=1715, outliers=400)
    Fs = np.concatenate([F[None], _hypotheses(rs, p, q, 300), rs.normal(size=(20, 3, 3)), np.zeros((1, 3, 3))])
    with Context(brief_pattern, levels=6, max_width=752, max_height=480) as c:
        for n in (1715, 1000, 33, 1, 0):
            counts, masks = c.ransac_score(Fs, p[:n], q[:n], 3.84, masks=True)
            ec, em = oracle.sampson_counts(Fs, p[:n], q[:n], 3.84)
            assert np.array_equal(counts, ec), n
            assert np.array_equal(masks, em), n
        assert counts.size == len(Fs)
        full = c.ransac_score(Fs, p, q)
        assert full[0] >= 1315 and full[-1] == 0


def test_ransac_score_on_matched_frames(brief_pattern):
    f0, f1 = synth.warped_pair(31)
    a, b = oracle.frame(f0, brief_pattern), oracle.frame(f1, brief_pattern)
    m = oracle.match(a[0], a[1], b[0], b[1], 752, 480)
    aoff = np.concatenate([[0], np.cumsum(a[1])])
    boff = np.concatenate([[0], np.cumsum(b[1])])
    scale = lambda l: np.prod([1.2] * int(l)) if l else 1.0
    p = np.array([[a[0][aoff[la] + ia]["x"] * scale(la), a[0][aoff[la] + ia]["y"] * scale(la)] for la, ia, _, _ in m])
    q = np.array([[b[0][boff[lb] + ib]["x"] * scale(lb), b[0][boff[lb] + ib]["y"] * scale(lb)] for _, _, lb, ib in m])
    Fs = _hypotheses(np.random.RandomState(2), p, q, 500)
    with Context(brief_pattern, levels=6, max_width=752, max_height=480) as c:
        counts = c.ransac_score(Fs, p, q)
    ec, _ = oracle.sampson_counts(Fs, p, q, 3.84)
    assert np.array_equal(counts, ec)
    assert counts.max() > len(m) // 4


@pytest.mark.parametrize("n_hyp,n", [(1, 1), (7, 31), (8, 32), (9, 257), (17, 256), (3, 5000)])
def test_binary32_decision_equals_binary64(n_hyp, n):
    """The scoring decides in binary32 where that is certain.  Hypotheses of
    every scale (also beyond binary32), points at the threshold, far outside
    the frame, infinite and not numbers: counts and masks equal the oracle's."""
    rs = np.random.RandomState(n_hyp * 1000 + n)
    pat = np.clip(np.rint(rs.normal(0, 6, (256, 4))), -13, 13).astype(np.int32)
    F, p, q = two_view(rs, n=n, outliers=n // 4)
    Fs = np.concatenate([F[None], _hypotheses(rs, p, q, n_hyp - 1)])[:n_hyp] if n >= 8 else rs.normal(size=(n_hyp, 3, 3))
    q = q.copy()
    q[::5] += rs.normal(0, 1.4, q[::5].shape)  # near the threshold
    p[-1:] = [[1e9, -3e7]]
    if n > 100:
        p[3], q[4], p[5] = [np.inf, 1.0], [np.nan, 2.0], [0.0, 0.0]
    with Context(pat, levels=6, max_width=752, max_height=480) as c:
        for scale in (1.0, 1e-4, 1e-9, 1e30, 1e-60, 1e150):
            for thr in (3.84, 1e-7, 1e9):
                counts, masks = c.ransac_score(Fs * scale, p, q, thr, masks=True)
                ec, em = oracle.sampson_counts(Fs * scale, p, q, thr)
                assert np.array_equal(counts, ec) and np.array_equal(masks, em), (scale, thr)


def test_binary32_decision_far_coordinates():
    """Coordinates far beyond any frame against matrix entries below
    binary32's range: what such an entry loses is no small part of its
    product.  Masks equal the oracle's, for pairs that a bound relative to
    the terms decides wrongly and for seeded ones over the whole range."""
    rs = np.random.RandomState(11)
    pat = np.clip(np.rint(rs.normal(0, 6, (256, 4))), -13, 13).astype(np.int32)
    cases = [
        ([5.19847117e-33, 2.86832077e-34, 0, 3.06804363e-47, 0, 1.35253869e-40, 6.74797655e-46, 1, -8.93523470e-09],
         [3.36596397e+35, 2.21408643e+01, 4.32841209e-12, 1.97015855e+24], 128632.39812623641),
        ([0, -4.21436813e-47, 0, 5.42532328e-29, 2.07247232e-22, -6.09367600e-20, 1, 2.79263952e-28, 2.31315755e-35],
         [-3.28058936e+06, 7.43869241e+30, 1.75687029e+35, 1.45843975e+02], 22942.1580560616),
        ([4.27588295e-38, 1.27277456e-02, -2.13807993e-45, -3.05614648e-46, -1.82482907e-20, -2.96136811e-48, 0, 1, 0],
         [-1.19746554e+35, -2.46484468e+00, 1.43011554e-10, 1.23084452e+15], 849.8911403708065),
    ]
    with Context(pat, levels=6, max_width=752, max_height=480) as c:
        for f, xy, thr in cases:
            args = np.array([f]), np.array([xy[:2]]), np.array([xy[2:]]), thr
            counts, masks = c.ransac_score(*args, masks=True)
            ec, em = oracle.sampson_counts(*args)
            assert np.array_equal(counts, ec) and np.array_equal(masks, em), (f, xy)
        Fs = rs.normal(size=(200, 9)) * 10.0 ** rs.uniform(-48, 0, (200, 9))
        Fs[np.arange(200), rs.randint(0, 9, 200)] = 1.0
        xy = rs.normal(size=(500, 4)) * 10.0 ** rs.uniform(-30, 37, (500, 4))
        for thr in (1e-5, 3.84, 1e5):
            counts, masks = c.ransac_score(Fs, xy[:, :2], xy[:, 2:], thr, masks=True)
            ec, em = oracle.sampson_counts(Fs, xy[:, :2], xy[:, 2:], thr)
            assert np.array_equal(counts, ec) and np.array_equal(masks, em), thr


def test_growing_calls_cost_no_allocation_each():
    """30 calls of ever more matches against 30 of the most: the kept staging
    grows a few times, not with every call (then they took 4.8 times as long,
    1.03 times without; the best of five contexts each)."""
    import time

    rs = np.random.RandomState(1)
    pat = np.clip(np.rint(rs.normal(0, 6, (256, 4))), -13, 13).astype(np.int32)
    Fs, p = rs.normal(size=(500, 3, 3)), rs.uniform(0, 700, (3000, 2))
    q = p + rs.normal(0, 3, p.shape)

    def run(sizes):
        with Context(pat, levels=6, max_width=752, max_height=480) as c:
            t0 = time.perf_counter()
            for n in sizes:
                c.ransac_score(Fs, p[:n], q[:n], masks=True)
            return time.perf_counter() - t0

    run([3000])
    growing, constant = min(run(range(100, 3001, 100)) for _ in range(5)), min(run([3000] * 30) for _ in range(5))
    assert growing < 2.0 * constant, (growing, constant)
