"""The blur cache is evaluated per run in the tiles that a test of a kept
keypoint can read (k_blur over the list of k_band_write).  Feature records
equal the oracle's where those tiles are few (frame caps, per-cell caps), for
patterns of a small and a large reach (beyond a tile row, 32), and at level
sizes around the tile's 64 x 32; the getter still returns the whole cache."""
import numpy as np
import pytest

import oracle
from uni_slam_gb300 import Batch, Context, synth

pytestmark = pytest.mark.gpu


def _pattern(reach: int) -> np.ndarray:
    p = np.random.RandomState(reach).randint(-reach, reach + 1, (256, 4)).astype(np.int32)
    p[0] = (reach, reach, -reach, -reach)
    return p


@pytest.mark.parametrize("size", [(64, 32), (65, 33), (63, 31), (130, 70), (37, 23), (257, 97), (512, 300)])
@pytest.mark.parametrize("reach,frame_cap,cell_cap", [(1, 0, 0), (13, 0, 0), (13, 40, 0), (13, 0, 2), (40, 0, 0), (40, 25, 1)])
def test_features_equal_oracle(size, reach, frame_cap, cell_cap):
    W, H = size
    pat = _pattern(reach)
    frames = list(synth.warped_pair(W + reach, W, H, n_rect=60, n_check=12, scale_by_area=False))
    levels = 3
    with Context(pat, levels=levels, max_width=W, max_height=H, cap_per_level=400, cell_cap=cell_cap,
                 frame_cap=frame_cap) as ctx:
        b = Batch(ctx, [(W, H)] * 2)
        try:
            b.process(frames)
            for i, f in enumerate(frames):
                exp, kept, raw = oracle.frame(f, pat, levels=levels, cap=400, cell_cap=cell_cap, frame_cap=frame_cap)
                got, gk, gr = b.features(i)
                assert np.array_equal(gk, kept) and np.array_equal(gr, raw)
                assert got.tobytes() == exp.tobytes()
                for l in range(levels):
                    want = oracle.blur_level(oracle.pyramid_level(f, l, levels))
                    assert np.array_equal(b.blur_level(i, l).view(np.uint32), want.view(np.uint32)), f"level {l}"
        finally:
            b.close()


def test_empty_and_refilled_lists():
    """Runs of one batch with no keypoint, many, then none again: the list is rebuilt by each run."""
    W, H = 200, 150
    pat = _pattern(13)
    full = synth.scene_frame(3, W, H)
    flat = np.full((H, W), 90, np.uint8)
    with Context(pat, levels=4, max_width=W, max_height=H) as ctx:
        b = Batch(ctx, [(W, H)])
        try:
            for f in (flat, full, flat, full[::-1].copy()):
                b.process([f])
                exp, kept, _ = oracle.frame(f, pat, levels=4)
                got, gk, _ = b.features(0)
                assert np.array_equal(gk, kept) and got.tobytes() == exp.tobytes()
        finally:
            b.close()
