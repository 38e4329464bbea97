"""The windowed matcher beside the sizes at which its lists, batches and emit
change: candidates of a batch (32) and of a quad (4), the caps at which the
number of bands changes, and features of a level beside a round of the emit
(8192).  Match lists against the oracle, alone and mixed in one batch."""
import numpy as np
import pytest

import oracle
from uni_slam_gb300 import Batch, Context, synth

pytestmark = pytest.mark.gpu

PATTERN = np.clip(np.rint(np.random.RandomState(5).normal(0, 6, (256, 4))), -13, 13).astype(np.int32)


def _check(frames, levels, cap, least, copies=1):
    h, w = frames[0].shape
    exp = [oracle.frame(f, PATTERN, levels=levels, cap=cap) for f in frames]
    distinct = [(0, 1), (1, 0)]
    pairs = distinct * copies
    lists = [oracle.match(exp[p][0], exp[p][1], exp[q][0], exp[q][1], w, h) for p, q in distinct]
    with Context(PATTERN, levels=levels, max_width=w, max_height=h, cap_per_level=cap) as c:
        b = Batch(c, [(w, h)] * 2, pairs)
        try:
            b.process(frames)
            for k in range(len(pairs)):
                m = b.matches(k)
                got = np.stack([m["lod_a"], m["idx_a"], m["lod_b"], m["idx_b"]], 1) if len(m) else np.zeros((0, 4), np.int32)
                want = lists[k % 2]
                assert np.array_equal(got, want), k
                assert len(want) >= least
        finally:
            b.close()


@pytest.mark.parametrize("cap", [1, 2, 3, 4, 5, 31, 32, 33, 63, 65])
@pytest.mark.parametrize("levels", [1, 3])
def test_partial_batches(cap, levels):
    _check(synth.warped_pair(41, 640, 480), levels, cap, 0)


@pytest.mark.parametrize("cap", [2500, 2501, 5001, 16001])
def test_caps_at_which_bands_change(cap):
    _check(synth.warped_pair(41, 640, 480), 2, cap, 500)


@pytest.mark.parametrize("cap", [8191, 8192, 8193])
def test_rounds_of_the_emit(cap):
    _check(synth.warped_pair(2024, 1920, 1080, n_rect=5000, n_check=500, scale_by_area=False), 2, cap, 500)


def test_accumulators_emptied_by_kept_features():
    """Caps far above what is kept (more than 64 MiB of accumulators)."""
    _check(synth.warped_pair(41, 320, 240), 6, 60000, 100, copies=4)
