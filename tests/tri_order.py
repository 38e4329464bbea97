"""Which of several tied pose candidates counts: the first in the order of the
cyclic decompositions (k_tri_gram's fallback), restated in numpy.  The order
follows from the signs that their rotations leave on the singular vectors."""
from __future__ import annotations

import numpy as np

from oracle import triangulate as T


def _angle(app, aqq, apq):
    """(cosine, sine) of the rotation that zeroes a_pq (|angle| <= 45 degrees)."""
    g = 100.0 * abs(apq)
    if abs(app) + g == abs(app) and abs(aqq) + g == abs(aqq):
        return 1.0, 0.0
    theta = (aqq - app) / (2.0 * apq)
    t = (1.0 if theta >= 0.0 else -1.0) / (abs(theta) + np.sqrt(theta * theta + 1.0))
    c = 1.0 / np.sqrt(t * t + 1.0)
    return c, t * c


def _rotate(a, v, pairs):
    """a = J^T a J, v = v J for disjoint rotations."""
    j = np.eye(len(a))
    for p, q in pairs:
        c, s = _angle(a[p, p], a[q, q], a[p, q])
        j[p, p] = j[q, q] = c
        j[p, q], j[q, p] = s, -s
    return j.T @ a @ j, v @ j


def _smallest9(a):
    """Eigenvector of the smallest eigenvalue: 9 rounds of 4 rotations a sweep (round robin around a tenth index)."""
    v = np.eye(9)
    for _ in range(12):
        for r in range(9):
            a, v = _rotate(a, v, [tuple(sorted(((r + k) % 9, (r + 9 - k) % 9))) for k in range(1, 5)])
    return v[:, np.argmin(np.diag(a))]


def _svd3(e):
    """(U, S, V) with det U = 1: V from E^T E by cyclic rotations, U's first two columns from E V."""
    a, v = e.T @ e, np.eye(3)
    for _ in range(15):
        for pair in ((0, 1), (0, 2), (1, 2)):
            a, v = _rotate(a, v, [pair])
    v = v[:, np.argsort(-np.diag(a), kind="stable")]
    ev = e @ v
    s = np.linalg.norm(ev, axis=0)
    u1 = ev[:, 0] / s[0]
    u2 = ev[:, 1] - (u1 @ ev[:, 1]) * u1
    u2 /= np.linalg.norm(u2)
    return np.stack([u1, u2, np.cross(u1, u2)], 1), s, v


def candidates(px, cam):
    """The four (R, t) of the rows px in the order of the decompositions."""
    prev, curr = (T.pixel_to_normalised(v, cam, 20, 1e-9) for v in (px[:, :2], px[:, 2:]))
    tp, tc = T.normalising_transform(prev), T.normalising_transform(curr)
    xp, yp = (prev @ tp[:2, :2].T + tp[:2, 2]).T
    xc, yc = (curr @ tc[:2, :2].T + tc[:2, 2]).T
    rows = np.stack([xc * xp, xc * yp, xc, yc * xp, yc * yp, yc, xp, yp, np.ones_like(xp)], 1)
    u, s, v = _svd3(_smallest9(rows.T @ rows).reshape(3, 3))
    mean = 0.5 * (s[0] + s[1])
    u, _, v = _svd3(tc.T @ (u @ np.diag([mean, mean, 0.0]) @ v.T) @ tp)
    if np.linalg.det(v) < 0.0:
        v[:, 2] *= -1.0
    w = np.array([[0.0, -1.0, 0.0], [1.0, 0.0, 0.0], [0.0, 0.0, 1.0]])
    r1, r2, t = u @ w @ v.T, u @ w.T @ v.T, u[:, 2]
    return [(r1, t), (r1, -t), (r2, t), (r2, -t)]
