"""Strips of the tile kernel vs the CPU oracle (needs a B200): one warp works on
4, 2 or 1 rows of a tile, chosen by the launch's tile count and configuration.
Images of every remainder against the strips (fewer rows or columns than one
strip, one more than a multiple), and every row count of every tile size in
every mode that launches it.  Images within 1e-4 and gradients within 1e-3
relative L2 (the reference's own tolerances); repeated steps, and the plain
path's, equal the batched step's up to the order of their float sums (1e-5)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import make_renderer, rel_l2

pytestmark = pytest.mark.gpu

GROUPS = ("d_vertices", "d_densities", "d_color_grads", "d_base_colors")


def _slot_groups(r, sc):
    """The fused step's gradient slots as the four groups of a backward pass."""
    s = r.grad_slots().cpu().numpy()[:20 * r.n_tets].reshape(-1, 20).astype(np.float64)
    dv = np.zeros((r.n_vertices, 3))
    np.add.at(dv, sc["indices"].reshape(-1, 4).ravel().astype(np.int64), s[:, 7:19].reshape(-1, 3))
    return {"d_vertices": dv.ravel(), "d_densities": s[:, 0], "d_base_colors": s[:, 1:4].ravel(),
            "d_color_grads": s[:, 4:7].ravel()}


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
    # the fused step's loss and gradients, each mode twice
    first = None
    for mode in ("batched", "plain") * 2:
        loss = r.accumulate_views([cam], [gt], mode=mode)
        np.testing.assert_allclose(loss, [want], rtol=1e-4)
        s = _slot_groups(r, sc)
        if first is None:
            first = (loss, s)
            for k in GROUPS:
                assert rel_l2(s[k], go[k]) <= 1e-3, k
        np.testing.assert_allclose(loss, first[0], rtol=1e-6)
        for k in GROUPS:
            assert rel_l2(s[k], first[1][k]) <= 1e-5, (mode, k)
    r.close()


@pytest.mark.parametrize("ts,threads", [(8, 0), (12, 0), (12, 320), (16, 0)])
@pytest.mark.parametrize("w,h", [(1, 1), (13, 5), (12, 12), (31, 3), (50, 37)])
def test_images_smaller_than_strips_and_remainders(c1_scene, oracle32, w, h, ts, threads):
    from rmesh_b200.camera import make_camera

    # a narrow field of view: a few tets over many pixels, so runs end inside rows
    _check(c1_scene, oracle32, make_camera((2.1, -1.9, 0.9), (0.0, 0.0, 0.0), 12.0, w, h), ts, threads)


def strip_view(ts, rows, fov=50.0):
    """A view, no multiple of the tile, whose adjoint takes ``rows`` rows per strip: one
    below 16 four-row strips per SM, four from six times as many (four times for 8-pixel
    tiles), two between."""
    import torch

    from rmesh_b200.camera import make_camera

    unit = 16 * torch.cuda.get_device_properties(0).multi_processor_count
    four = 4 if ts == 8 else 6
    k = int(np.ceil(np.sqrt({1: 0.3, 2: 1.1, 4: four}[rows] * unit / (ts // 4))))
    strips = k * k * (ts // 4)
    assert rows == (1 if strips < unit else 2 if strips < four * unit else 4)
    return make_camera((2.1, -1.9, 0.9), (0.0, 0.0, 0.0), fov, k * ts - 1, k * ts - 3)


# forwards of the same sizes take 1, 2 and 2 rows; a wide configuration takes 2 for 4
@pytest.mark.parametrize("ts,threads,rows", [(8, 0, 1), (8, 0, 2), (8, 0, 4), (8, 128, 4), (12, 0, 1), (12, 0, 2),
                                             (12, 0, 4), (12, 320, 4), (16, 0, 1), (16, 0, 2), (16, 0, 4), (16, 512, 4)])
def test_every_row_count(c1_scene, oracle32, ts, threads, rows):
    _check(c1_scene, oracle32, strip_view(ts, rows), ts, threads)


# 12-pixel tiles on 148 SMs: 784x777 is 4,290 tiles (two rows for the adjoint), 1000x993
# 6,972 (four)
@pytest.mark.parametrize("size,threads", [(784, 0), (1000, 0), (1000, 320)])
def test_both_sides_of_the_strip_rule(c1_scene, oracle32, size, threads):
    from rmesh_b200.camera import make_camera

    _check(c1_scene, oracle32, make_camera((2.1, -1.9, 0.9), (0.0, 0.0, 0.0), 50.0, size, size - 7), 12, threads)


@pytest.mark.parametrize("rows", [1, 2])
@pytest.mark.parametrize("ts", [8, 12, 16])
def test_error_statistics_of_every_row_count(c1_scene, oracle32, ts, rows):
    """The statistics against the oracle as in test_gpu_error.py, at launches of one- and
    two-row strips of each tile size."""
    cam = strip_view(ts, rows)
    n = cam.width * cam.height
    r = make_renderer(c1_scene, cam, tile_size=ts)
    r.forward_tiled(cam.cam_pos, cam.vp, cam.c2w_intrinsics)
    rng = np.random.default_rng(ts + rows)
    pe, se = rng.uniform(0, 1, n).astype(np.float32), rng.uniform(0, 1, n).astype(np.float32)
    err, cnt = r.forward_error(pe, se)
    ref = oracle32.forward_tiled(c1_scene, cam, tile_size=ts)
    e_ref, c_ref = oracle32.error_stats(c1_scene, cam, ref, pe, se, tile_size=ts)
    for k in (0, 1, 2, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15):
        assert rel_l2(err[:, k], e_ref[:, k]) <= 1e-4, k
    assert np.all(err[:, 3:5] == 0.0)
    assert np.abs(cnt[:, 0] - c_ref[:, 0]).sum() <= max(2, c_ref[:, 0].sum() // 10000)
    assert np.all(np.abs(cnt[:, 1] - c_ref[:, 1]) <= np.maximum(2, c_ref[:, 1] // 10000))
    r.close()


@pytest.mark.parametrize("ts,rows,aux_dim", [(8, 2, 2), (8, 4, 2), (12, 2, 2), (12, 4, 2), (16, 2, 2), (16, 4, 2),
                                             (12, 1, 9), (8, 2, 13), (16, 1, 64)])
def test_aux_channels_of_every_row_count(c1_scene, oracle32, ts, rows, aux_dim):
    """Aux images and all gradients through them; more than 8 channels leave shared
    memory (kAuxShared) for the output rows."""
    from rmesh_b200 import RMeshRenderer

    sc, cam = c1_scene, strip_view(ts, rows)
    rng = np.random.default_rng(aux_dim)
    ad = rng.uniform(-1, 1, aux_dim * sc["densities"].size).astype(np.float32)
    r = RMeshRenderer(sc["vertices"], sc["indices"], sc["base_colors"], sc["densities"], sc["color_grads"],
                      sc["circumdata"], cam.width, cam.height, aux_dim=aux_dim, tile_size=ts)
    r.set_aux_data(ad)
    img, aux = r.forward_tiled(cam.cam_pos, cam.vp, cam.c2w_intrinsics, render_aux=True)
    ref = oracle32.forward_tiled(sc, cam, tile_size=ts, aux=True, aux_data=ad)
    assert np.abs(img - ref["image"]).max() <= 1e-4
    assert np.abs(aux[..., 8:] - ref["aux"][..., 8:]).max() <= 1e-4
    gt = rng.uniform(0, 1, (cam.height, cam.width, 3)).astype(np.float32)
    _, dl = oracle32.loss(ref["image"], gt, 1)
    dl_aux = rng.normal(0, 1.0 / (cam.width * cam.height), (cam.height, cam.width, aux_dim)).astype(np.float32)
    g = r.backward(dl, dl_aux)
    go = oracle32.backward(sc, cam, dl, ref, tile_size=ts, threads=oracle32.max_threads, aux_data=ad, dl_aux=dl_aux)
    for k in GROUPS + ("d_aux_data",):
        assert rel_l2(g[k], go[k]) <= 1e-3, k
    r.close()


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
