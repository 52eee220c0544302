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


def _one_tet(v, density, color, grad):
    from rmesh_b200.scenes import circumspheres

    v = np.asarray(v, np.float32).ravel()
    idx = np.arange(4, dtype=np.uint32)
    return {"vertices": v, "indices": idx, "base_colors": np.asarray(color, np.float32),
            "densities": np.array([density], np.float32), "color_grads": np.asarray(grad, np.float32),
            "circumdata": circumspheres(v, idx)}


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


def test_optical_depth_derivative_is_one_quotient():
    """A tet crossed over exactly 2 units, its colour 1 at the entry and clipped to 0 at
    the exit: the density's gradient is -2 dphi(od) and, at these depths, dphi = -1 / od^2
    to the last bit.  Its errors are the rounding of od^2 (rms 0.4 units) and one fast
    quotient's (0.4 were it correctly rounded); 0.8 together leaves that quotient 0.7."""
    from rmesh_b200.camera import make_camera

    v = ((-4, 0, -3), (4, 0, -3), (0, 0, 9), (0, 4, 3))
    cam = make_camera((0.0, -4.0, 0.0), (0.0, 0.0, 0.0), 60.0, 1, 1)
    r = make_renderer(_one_tet(v, 1.0, (1.0, 0.5, 0.5), (0.0, -1.0, 0.0)), cam)
    p = r.get_params()
    dl = np.array([[[1.0, 0.0, 0.0, 0.0]]], np.float32)
    err = []
    for d in np.random.default_rng(5).uniform(23.5, 43.5, 1500).astype(np.float32):
        r.update_params(p["vertices"], p["base_colors"], np.array([d], np.float32), p["color_grads"])
        r.forward_tiled(cam.cam_pos, cam.vp, cam.c2w_intrinsics)
        g = r.backward(dl)["d_densities"][0]
        od = 2.0 * float(d)
        want = -2.0 * (np.exp(-od) * (od + 1.0) - 1.0) / od ** 2
        err.append((float(g) - want) / want)
    r.close()
    err = np.array(err) / UNIT
    # (__fdividef: two units in the last place, four of these)
    assert np.abs(err).max() <= 1.0 + 4.0
    assert np.sqrt((err ** 2).mean()) <= 0.8


def test_aux_gradient_of_an_almost_opaque_tet():
    """At od 87.4..87.9 alpha's derivative e^-od is below 2^-126, the smallest normal
    number, and still the whole of the density's gradient when only an aux channel has
    a loss.  e^-od rounds the exponent od log2(e), about 126, to 2^-18."""
    from rmesh_b200 import RMeshRenderer
    from rmesh_b200.camera import make_camera

    v = ((-4, 0, -3), (4, 0, -3), (0, 0, 9), (0, 4, 3))
    cam = make_camera((0.0, -4.0, 0.0), (0.0, 0.0, 0.0), 60.0, 1, 1)
    for d in (43.7, 43.8, 43.95):
        sc = _one_tet(v, d, (1.0, 0.5, 0.5), (0.0, 0.0, 0.0))
        r = RMeshRenderer(sc["vertices"], sc["indices"], sc["base_colors"], sc["densities"], sc["color_grads"],
                          sc["circumdata"], 1, 1, 1)
        r.set_aux_data(np.ones(1, np.float32))
        r.forward_tiled(cam.cam_pos, cam.vp, cam.c2w_intrinsics, render_aux=True)
        g = r.backward(np.zeros((1, 1, 4), np.float32), np.full((1, 1, 1), 1e30, np.float32))
        r.close()
        want = 2.0 * np.exp(-2.0 * float(np.float32(d))) * 1e30
        np.testing.assert_allclose(g["d_densities"][0], want, rtol=4 * 2.0 ** -18)
