"""Rigid motion of the object per view, composed into projection matrices.

theta = (tx, ty, tz, rx, ry, rz): a translation in mm and rotations in degrees
about the volume's x, y, z axes.  A voxel at X in the reconstruction frame
sits at M(theta) X = R X + t during the view, R = Rz Ry Rx, so the view's
projection matrix becomes P(theta) = P0 M(theta).  Composition and the
derivatives dP/dtheta_j are computed in FP64 on the host.
"""
from __future__ import annotations

import numpy as np

_DEG = np.pi / 180.0


def _rot(axis: int, a: np.ndarray):
    """Rotations about an axis by the angles a (n,), and their derivatives: (n, 3, 3) each."""
    c, s = np.cos(a), np.sin(a)
    r, dr = np.zeros((len(a), 3, 3)), np.zeros((len(a), 3, 3))
    r[:, axis, axis] = 1.0
    i, j = [(1, 2), (0, 2), (0, 1)][axis]
    sign = -1.0 if axis == 1 else 1.0   # y: [[c, 0, s], [0, 1, 0], [-s, 0, c]]
    r[:, i, i], r[:, j, j], r[:, i, j], r[:, j, i] = c, c, -sign * s, sign * s
    dr[:, i, i], dr[:, j, j], dr[:, i, j], dr[:, j, i] = -s, -s, -sign * c, sign * c
    return r, dr


def _rigid_all(theta: np.ndarray, derivatives: bool = True):
    """M(theta_v) (n, 4, 4) and dM/dtheta_j (n, 6, 4, 4), FP64, all views at
    once: one view at a time the two passes over 360 views took 19 ms of a
    gradient step whose kernels take 55 (0.4 ms now)."""
    t = np.asarray(theta, np.float64).reshape(-1, 6)
    (rx, drx), (ry, dry), (rz, drz) = (_rot(k, t[:, 3 + k] * _DEG) for k in range(3))
    M = np.zeros((len(t), 4, 4))
    M[:, :3, :3] = rz @ ry @ rx
    M[:, :3, 3] = t[:, :3]
    M[:, 3, 3] = 1.0
    if not derivatives:
        return M, None
    dM = np.zeros((len(t), 6, 4, 4))
    for j in range(3):
        dM[:, j, j, 3] = 1.0
    dM[:, 3, :3, :3] = rz @ ry @ drx * _DEG
    dM[:, 4, :3, :3] = rz @ dry @ rx * _DEG
    dM[:, 5, :3, :3] = drz @ ry @ rx * _DEG
    return M, dM


def rigid(theta) -> tuple[np.ndarray, np.ndarray]:
    """M(theta) (4 x 4) and dM/dtheta_j (6 x 4 x 4), FP64, of one motion (what
    follows its six parameters is not read)."""
    t = np.asarray(theta, np.float64)
    if t.ndim == 0 or len(t) < 6:
        raise IndexError(f"a motion has six parameters, got shape {t.shape}")
    if t.ndim != 1:
        raise ValueError(f"rigid takes one motion, got shape {t.shape}")
    M, dM = _rigid_all(t[:6])
    return M[0], dM[0]


def _views(P0, theta):
    """P0 (n, 3, 4) and the motions of its views (a theta of more views is cut)."""
    P0 = np.asarray(P0, np.float64).reshape(-1, 3, 4)
    th = np.asarray(theta, np.float64).reshape(-1, 6)
    if not len(P0):
        raise ValueError("no projection matrices")
    if len(th) < len(P0):
        raise IndexError(f"{len(th)} motions for {len(P0)} views")
    return P0, th[:len(P0)]


def moved_ptms(P0, theta) -> np.ndarray:
    """P0 M(theta_v) per view: (n, 12) FP64."""
    P0, th = _views(P0, theta)
    return (P0 @ _rigid_all(th, derivatives=False)[0]).reshape(-1, 12)


def ptm_derivatives(P0, theta) -> np.ndarray:
    """dP/dtheta_j = P0 dM/dtheta_j per view: (n, 6, 12) FP64."""
    P0, th = _views(P0, theta)
    return (P0[:, None] @ _rigid_all(th)[1]).reshape(-1, 6, 12)


def seeded_motion(n_views: int, seed: int, shift_mm: float = 0.5, rot_deg: float = 0.3) -> np.ndarray:
    """(n, 6) motion, uniform in +/- shift_mm and +/- rot_deg."""
    rng = np.random.default_rng(seed)
    th = np.empty((n_views, 6))
    th[:, :3] = rng.uniform(-shift_mm, shift_mm, (n_views, 3))
    th[:, 3:] = rng.uniform(-rot_deg, rot_deg, (n_views, 3))
    return th
