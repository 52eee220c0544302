"""Roundings of the tile kernel's per-crossing arithmetic, seen through single tets
whose geometry is exact in 32 bits (needs a B200).  Errors are relative, in units
of 2^-24: half a unit in the last place of a number just above a power of two."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import make_renderer

pytestmark = pytest.mark.gpu

UNIT = 2.0 ** -24
FACES = ((0, 2, 1, 3), (1, 2, 3, 0), (0, 3, 2, 1), (3, 0, 1, 2))


def test_entry_normal_is_correctly_rounded():
    """2,000 opaque tets with integer vertices, so that the face normals are exact and
    the weight of a pixel inside one is exactly 1: the aux image holds the unit normal
    after two roundings, the square root and the division."""
    from rmesh_b200.camera import make_camera
    from rmesh_b200.scenes import circumspheres

    rng = np.random.default_rng(3)
    at = 32.0 * np.stack(np.meshgrid(np.arange(-22, 23), np.arange(-22, 23)), -1).reshape(-1, 2)
    v = rng.integers(-12, 13, (at.shape[0], 4, 3)).astype(np.float64)
    v[:, :, 0] += at[:, None, 0]
    v[:, :, 1] += at[:, None, 1]
    v = v[np.abs(np.linalg.det(v[:, 1:] - v[:, :1])) > 500]
    m = v.shape[0]
    vert, idx = v.astype(np.float32).ravel(), np.arange(4 * m, dtype=np.uint32)
    sc = {"vertices": vert, "indices": idx, "base_colors": np.full(3 * m, 0.5, np.float32),
          "densities": np.full(m, 30.0, np.float32), "color_grads": np.zeros(3 * m, np.float32),
          "circumdata": circumspheres(vert, idx)}
    cam = make_camera((60.0, -90.0, 2000.0), (0.0, 0.0, 0.0), 42.0, 1000, 1000, near=1.0, far=4000.0)
    r = make_renderer(sc, cam)
    _, aux = r.forward_tiled(cam.cam_pos, cam.vp, cam.c2w_intrinsics, render_aux=True)
    r.close()
    aux = aux.reshape(-1, 8)
    got = np.unique(aux[aux[:, 4] == 1.0, :3], axis=0).astype(np.float64)
    n = []
    for a, b, c, o in FACES:
        q = np.cross(v[:, c] - v[:, a], v[:, b] - v[:, a])
        out = np.where((q * (v[:, o] - v[:, a])).sum(1, keepdims=True) < 0, 1.0, -1.0)
        n.append(out * q / np.linalg.norm(q, axis=1, keepdims=True))
    n = np.concatenate(n)
    want = n[np.argmax(got @ n.T, axis=1)]
    near = np.abs(got - want).max(1) < 1e-6  # pixels of one tet only
    assert near.sum() > 2000
    got, want = got[near], want[near]
    assert np.all(got[want == 0.0] == 0.0)
    err = np.abs(got - want)[want != 0.0] / np.abs(want[want != 0.0])
    assert err.max() <= 2.001 * UNIT
