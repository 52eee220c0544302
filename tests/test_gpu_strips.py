"""Strips of the tile kernel vs the CPU oracle (needs a B200): one warp works on
4, 2 or 1 rows of a tile, chosen by the launch's tile count and configuration.
Images of every remainder against the strips (fewer rows or columns than one
strip, one more than a multiple) and launches on both sides of the rule, with
images within 1e-4 and gradients within 1e-3 relative L2 (the reference's own
tolerances) and repeated steps equal to the plain path's."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import make_renderer, rel_l2

pytestmark = pytest.mark.gpu

GROUPS = ("d_vertices", "d_densities", "d_color_grads", "d_base_colors")


def _check(sc, oracle, cam, ts, threads):
    r = make_renderer(sc, cam, tile_size=ts)
    r.set_tile_config(ts, threads)
    img = r.forward_tiled(cam.cam_pos, cam.vp, cam.c2w_intrinsics)
    ref = oracle.forward_tiled(sc, cam, tile_size=ts)
    assert np.abs(img - ref["image"]).max() <= 1e-4
    gt = np.random.default_rng(ts).uniform(0, 1, (cam.height, cam.width, 3)).astype(np.float32)
    want, dl = oracle.loss(ref["image"], gt, 1)
    go = oracle.backward(sc, cam, dl, ref, tile_size=ts, threads=oracle.max_threads)
    g = r.backward(dl)
    for k in GROUPS:
        assert rel_l2(g[k], go[k]) <= 1e-3, k
    # the fused step's loss and gradients (the slots' vertex sums against the oracle's)
    for mode in ("batched", "plain"):
        loss = r.accumulate_views([cam], [gt], mode=mode)
        np.testing.assert_allclose(loss, [want], rtol=1e-4)
        slots = r.grad_slots().cpu().numpy()[:20 * r.n_tets].reshape(-1, 20)
        assert rel_l2(slots[:, 0], go["d_densities"]) <= 1e-3
        assert rel_l2(slots[:, 4:7].ravel(), go["d_color_grads"]) <= 1e-3
    r.close()


@pytest.mark.parametrize("ts,threads", [(8, 0), (12, 0), (12, 320), (16, 0)])
@pytest.mark.parametrize("w,h", [(1, 1), (13, 5), (12, 12), (31, 3), (50, 37)])
def test_images_smaller_than_strips_and_remainders(c1_scene, oracle32, w, h, ts, threads):
    from rmesh_b200.camera import make_camera

    # a narrow field of view: a few tets over many pixels, so runs end inside rows
    _check(c1_scene, oracle32, make_camera((2.1, -1.9, 0.9), (0.0, 0.0, 0.0), 12.0, w, h), ts, threads)


# 12-pixel tiles: 784 px is 4356 tiles (thin strips), 1000 px 7056 (four rows for the adjoint on 148 SMs)
@pytest.mark.parametrize("size,threads", [(784, 0), (1000, 0), (1000, 320)])
def test_both_sides_of_the_strip_rule(c1_scene, oracle32, size, threads):
    from rmesh_b200.camera import make_camera

    _check(c1_scene, oracle32, make_camera((2.1, -1.9, 0.9), (0.0, 0.0, 0.0), 50.0, size, size - 7), 12, threads)


@pytest.mark.parametrize("n", [1, 4, 8, 16])
def test_batched_views_equal_single_views(c1_scene, n):
    """Batched runs split emission groups over 8, 4, 2 or 1 blocks, gather their
    tet records in a kernel of their own (n > 1) and skip the adjoint's spans; each
    image equals the single-view forward's bit for bit."""
    from rmesh_b200.camera import orbit_cameras

    cams = orbit_cameras(n, seed=5, radius=(2.2, 3.4), resolutions=((96, 80),))
    r = make_renderer(c1_scene, cams[0])
    imgs = r.forward_views(cams)
    for c, img in zip(cams, imgs):
        np.testing.assert_array_equal(img, r.forward_tiled(c.cam_pos, c.vp, c.c2w_intrinsics))
    r.close()
