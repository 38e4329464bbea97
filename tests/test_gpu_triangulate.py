"""Batched two-view triangulation on the GPU (uslam_triangulate,
uslam_pixel_to_normalised) against the reference's own TriangulateCPU
(golden vectors from triangulate_cpu.cpp) and the oracle restatement, with
the tolerances stated in test_oracle_triangulate.py: rays bit-exact, pose
1e-9, landmarks 1e-8 x max(1, |z|), counts and keep masks exact."""
import os

import numpy as np
import pytest

from oracle import triangulate as T
from tri_check import case_opts, check_against_reference
from tri_order import candidates
from uni_slam_gb300 import Context, USlamError, synth

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "triangulate_cases.npz")


@pytest.fixture(scope="module")
def ctx(brief_pattern):
    with Context(brief_pattern, levels=6, max_width=752, max_height=480) as c:
        yield c


def test_rays_bit_exact(ctx):
    g = np.load(GOLDEN)
    rays = ctx.pixel_to_normalised(g["undistort/px"], g["undistort/cam"], 20, 1e-9)
    assert np.array_equal(rays.view(np.uint64), g["undistort/rays"].view(np.uint64))
    # every pixel of two of the golden scenes, both views, other iteration limits
    for name in ("mixed_800", "two_undistort_iters"):
        rows, cam, o = g[f"{name}/rows"], g[f"{name}/cam"], case_opts(g[f"{name}/opts"])
        px = rows[:, 1:5].astype(np.float64).reshape(-1, 2)
        want = T.pixel_to_normalised(px, cam, o["undistort_iterations"], o["undistort_tolerance"])
        got = ctx.pixel_to_normalised(px, cam, o["undistort_iterations"], o["undistort_tolerance"])
        assert np.array_equal(got.view(np.uint64), want.view(np.uint64)), name


def test_golden_cases_batched(ctx):
    """All golden scenes in as few calls as their options allow (one call per
    distinct option set), each pair against the reference's result."""
    g = np.load(GOLDEN)
    names = sorted({k.split("/")[0] for k in g.files if not k.startswith("undistort/")})
    groups = {}
    for name in names:
        groups.setdefault(tuple(g[f"{name}/opts"]), []).append(name)
    for opts, group in groups.items():
        o = case_opts(np.array(opts))
        cam = g[f"{group[0]}/cam"]
        assert all(np.array_equal(g[f"{n}/cam"], cam) for n in group)
        res = ctx.triangulate([g[f"{n}/rows"][:, 1:5].astype(np.float64) for n in group], cam, o)
        for name, r in zip(group, res):
            check_against_reference(r, g[f"{name}/pose"], g[f"{name}/stats"], g[f"{name}/keep"],
                                    g[f"{name}/landmarks"], name)


def test_many_pairs_against_oracle(ctx):
    """24 seeded scenes of mixed sizes (including empty, 7-row and 8-row
    pairs) in one call, each against the oracle."""
    parts, cam = [], synth.SCENE_CAMERA
    sizes = [1500, 0, 7, 8, 33, 640, 1200, 300] * 3
    for k, n in enumerate(sizes):
        rows, _, _, _ = synth.two_view_scene(seed=500 + k, n=max(n, 1), outlier_frac=0.01 * (k % 3),
                                             rot_sigma=0.01 + 0.01 * (k % 4))
        parts.append(rows[:n, 1:5].astype(np.float64))
    res = ctx.triangulate(parts, cam)
    assert len(res) == len(parts)
    for k, (px, r) in enumerate(zip(parts, res)):
        want = T.triangulate(px, cam)
        pose = np.concatenate([want["rotation"].ravel(), want["translation"]])
        stats = [want["input_matches"], want["landmark_count"], want["cheirality_passes"],
                 want["mean_reprojection_error_px"], want["pose_recovered"], want["rotation_angle_rad"]]
        check_against_reference(r, pose, stats, want["keep"], want["landmarks"], f"pair {k} n={len(px)}")


def test_deterministic_and_single_pair(ctx):
    rows, cam, _, _ = synth.two_view_scene(seed=77, n=1000, outlier_frac=0.01)
    px = rows[:, 1:5].astype(np.float64)
    a = ctx.triangulate(px, cam)
    b = ctx.triangulate([px, px], cam)
    for r in b:
        assert np.array_equal(r["landmarks"].view(np.uint64), a["landmarks"].view(np.uint64))
        assert np.array_equal(r["rotation"].view(np.uint64), a["rotation"].view(np.uint64))
        assert r["landmark_count"] == a["landmark_count"]


def test_edge_calls(ctx):
    cam = synth.SCENE_CAMERA
    assert ctx.triangulate([], cam) == []
    r = ctx.triangulate(np.zeros((5, 4)), cam)
    assert r["input_matches"] == 5 and r["landmark_count"] == 0 and not r["pose_recovered"]
    assert np.array_equal(r["rotation"], np.eye(3))
    with pytest.raises(USlamError):
        ctx.triangulate(np.zeros((10, 4)), cam, {"min_inliers": 4})
    assert ctx.pixel_to_normalised(np.zeros((0, 2)), cam).shape == (0, 2)


@pytest.fixture(scope="module")
def own_ctx():
    pat = np.clip(np.rint(np.random.RandomState(5).normal(0, 6, (256, 4))), -13, 13).astype(np.int32)
    with Context(pat, max_width=752, max_height=480) as c:
        yield c


@pytest.mark.parametrize("n", [16, 31, 32, 33, 63, 64, 65, 1023, 1025, 2500])
@pytest.mark.parametrize("noise", [0.0, 0.3])
def test_edges_of_chunks_and_methods(own_ctx, n, noise):
    """Row counts beside a chunk (32 rows), the 9-vector's two methods (64
    rows) and 32 chunks, with and without a gap below the smallest singular
    value, alone and as one of three pairs, against the oracle."""
    px = synth.two_view_scene(seed=900 + n, n=n, noise_px=noise)[0][:, 1:5].astype(np.float64)
    want = T.triangulate(px, synth.SCENE_CAMERA)
    pose = np.concatenate([want["rotation"].ravel(), want["translation"]])
    stats = [want["input_matches"], want["landmark_count"], want["cheirality_passes"],
             want["mean_reprojection_error_px"], want["pose_recovered"], want["rotation_angle_rad"]]
    one = own_ctx.triangulate(px, synth.SCENE_CAMERA)
    for r in [one] + own_ctx.triangulate([px[:9], px, px[:8]], synth.SCENE_CAMERA)[1:2]:
        check_against_reference(r, pose, stats, want["keep"], want["landmarks"], f"n={n} noise={noise}")


@pytest.mark.parametrize("seed", [6, 12, 37])
def test_tied_candidates(own_ctx, seed):
    """Unrelated pixels, several candidates with the most points: one of them
    is the result, the same one alone and among other pairs."""
    px = np.random.RandomState(seed).uniform([20, 20, 20, 20], [700, 440, 700, 440], (12, 4))
    want = T.triangulate(px, synth.SCENE_CAMERA)
    top = np.flatnonzero(want["in_front"] == want["in_front"].max())
    assert len(top) > 1
    rays = [T.pixel_to_normalised(v, synth.SCENE_CAMERA, 20, 1e-9) for v in (px[:, :2], px[:, 2:])]
    cands = T.decompose_essential(T.fit_essential(*rays))
    one = own_ctx.triangulate(px, synth.SCENE_CAMERA)
    two = own_ctx.triangulate([px[::-1].copy(), px], synth.SCENE_CAMERA)[1]
    assert one["cheirality_passes"] == want["in_front"].max()
    assert min(np.abs(one["rotation"] - cands[k][0]).max() + np.abs(one["translation"] - cands[k][1]).max()
               for k in top) <= 1e-9
    assert np.array_equal(one["rotation"], two["rotation"]) and np.array_equal(one["translation"], two["translation"])


def _plane_rows(seed, n, cam):
    """Rows of a plane seen from two poses, exact to rounding: the 8-point
    system has rank 6."""
    rs = np.random.RandomState(seed)
    xy = rs.uniform(-0.5, 0.5, (n, 2))
    q = np.c_[xy, np.ones(n)] @ (np.eye(3) + rs.normal(0, 0.05, (3, 3))).T
    q = q[:, :2] / q[:, 2:]
    return np.c_[xy * cam[:2] + cam[2:4], q * cam[:2] + cam[2:4]]


@pytest.mark.parametrize("n", [64, 65, 640])
@pytest.mark.parametrize("scene", ["plane", "seven", "point"])
def test_rank_deficient_systems(own_ctx, scene, n):
    """64 rows or more whose 8-point system has a small pivot before its last
    (a plane; seven distinct rows; one): the whole CTA goes over to the cyclic
    method.  The essential matrix is not determined, but it is one: the result
    is a rotation, the same bits on repeated calls and among other pairs."""
    cam = np.array([458.0, 457.0, 367.0, 248.0, 0.0, 0.0, 0.0, 0.0])
    px = _plane_rows(n, n, cam)
    if scene != "plane":
        px = px[np.arange(n) % (7 if scene == "seven" else 1)]
    full = synth.two_view_scene(seed=41, n=200, cam=cam)[0][:, 1:5].astype(np.float64)
    one = own_ctx.triangulate(px, cam)
    again = [own_ctx.triangulate(px, cam)] + own_ctx.triangulate([full, px, px, full[:9]], cam)[1:3]
    r = one["rotation"]
    assert np.abs(r @ r.T - np.eye(3)).max() <= 1e-9 and abs(np.linalg.det(r) - 1.0) <= 1e-9
    for a in again:
        for key in ("rotation", "translation", "landmarks"):
            assert np.array_equal(a[key].view(np.uint64), one[key].view(np.uint64)), key
        assert a["cheirality_passes"] == one["cheirality_passes"] and np.array_equal(a["keep"], one["keep"])


@pytest.mark.parametrize("n", [64, 97, 256])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_close_smallest_eigenvalues(own_ctx, n, seed):
    """Unrelated pixels: the ratio of the two smallest eigenvalues of the 8-point
    system lies between 0.47 and 0.75, on both sides of where the squared
    inverse settles (about 0.6); beyond it the cyclic method decides.  The pose equals one of the oracle's best candidates."""
    px = np.random.RandomState(1000 * seed + n).uniform([20, 20, 20, 20], [700, 440, 700, 440], (n, 4))
    want = T.triangulate(px, synth.SCENE_CAMERA)
    rays = [T.pixel_to_normalised(v, synth.SCENE_CAMERA, 20, 1e-9) for v in (px[:, :2], px[:, 2:])]
    cands = T.decompose_essential(T.fit_essential(*rays))
    got = own_ctx.triangulate(px, synth.SCENE_CAMERA)
    assert got["cheirality_passes"] == want["in_front"].max()
    assert min(np.abs(got["rotation"] - cands[k][0]).max() + np.abs(got["translation"] - cands[k][1]).max()
               for k in np.flatnonzero(want["in_front"] == want["in_front"].max())) <= 1e-9


@pytest.mark.parametrize("n", [20, 80])
@pytest.mark.parametrize("prev,curr", [(1.0, 1e19), (1.0, 1e20), (1.0, 1e21), (1.0, 1e22), (1e3, 1e21)])
def test_spreads_beyond_binary32(own_ctx, n, prev, curr):
    """Current points spread so far that squares of the pose's lengths leave
    binary32's range.  No 64-bit method can tell the pose of such rows, but
    they have one: a rotation and a direction of length 1, and as a generic
    row is in front of both cameras for one of the four candidates, the best
    of them has points."""
    cam = np.array([458.0, 457.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0])
    for seed in range(8):
        px = np.random.RandomState(seed).normal(0, 300, (n, 4)) * [prev, prev, curr, curr]
        r = own_ctx.triangulate(px, cam)
        rot = r["rotation"]
        assert r["cheirality_passes"] > 0, seed
        assert np.abs(rot @ rot.T - np.eye(3)).max() <= 1e-9 and abs(np.linalg.det(rot) - 1.0) <= 1e-9, seed
        assert abs(np.linalg.norm(r["translation"]) - 1.0) <= 1e-9, seed


@pytest.mark.parametrize("n,seed", [(8, 18), (8, 384), (9, 23), (9, 214), (10, 0), (10, 381), (12, 10), (12, 135), (14, 5),
                                    (14, 328), (70, 134), (80, 2), (80, 362)])
def test_tie_goes_to_first_decomposed(own_ctx, n, seed):
    """Of the candidates that tie for the most points the first in the order
    of the cyclic decompositions counts.  In these scenes the order in which
    the faster methods hold the candidates has another one of them first."""
    px = np.random.RandomState(seed * 20 + n).uniform([20, 20, 20, 20], [700, 440, 700, 440], (n, 4))
    want = T.triangulate(px, synth.SCENE_CAMERA)
    top = want["in_front"].max()
    assert np.count_nonzero(want["in_front"] == top) > 1
    rays = [T.pixel_to_normalised(v, synth.SCENE_CAMERA, 20, 1e-9) for v in (px[:, :2], px[:, 2:])]
    plain = T.decompose_essential(T.fit_essential(*rays))  # in_front's order
    for rot, t in candidates(px, synth.SCENE_CAMERA):
        k = int(np.argmin([np.abs(rot - a).max() + np.abs(t - b).max() for a, b in plain]))
        if want["in_front"][k] == top:
            break
    got = own_ctx.triangulate(px, synth.SCENE_CAMERA)
    assert got["cheirality_passes"] == top
    np.testing.assert_allclose(got["rotation"], rot, rtol=0, atol=1e-9)
    np.testing.assert_allclose(got["translation"], t, rtol=0, atol=1e-9)
