"""Workloads of the renderer through its public entry points, from one small
preview image to the sixteen-view training step.

Each case is a plain dict:

  path    the entry point (see ``run``)
  cloud   mesh: "uniform" or "gmm" (Delaunay of ``points`` seeded points in the
          style of the benchmark configurations) or "grid" (``points`` cells per
          axis, five tets per cell, jittered vertices)
  sh      SH degree of the colours, -1 for base colours
  width, height, views
          image sizes; ``width`` 0 draws each view's size from the mixed set of
          the batched benchmark configuration
  inside  the camera stands inside the mesh (a viewer flying through a scene)
  aux     custom auxiliary channels per tet
  targets "host" or "device": where a training step's target images are

The mesh of a size is built once per process and turned by a random rotation
per seed (Delaunay stays Delaunay); colours, densities, cameras, targets and
gradients are drawn anew for each seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from rmesh_b200 import RMeshModule, RMeshRenderer
from rmesh_b200.camera import make_camera, orbit_cameras
from rmesh_b200.scenes import delaunay_tets, gmm_cloud, uniform_cloud

MIXED = ((256, 256), (512, 512), (800, 600), (1024, 1024))
# learning rates of a late training stage: small enough that a few passes over
# one state stay comparable
LR = dict(lr_verts=1e-6, lr_dens=1e-5, lr_grads=1e-6)
LR_SH = 1e-5


def _case(name, path, cloud, points, sh, width, height, views=1, inside=False, aux=0, targets="device"):
    return dict(name=name, path=path, cloud=cloud, points=points, sh=sh, width=width, height=height, views=views,
                inside=inside, aux=aux, targets=targets)


def listed():
    return [
        # smallest call: one preview image of a small mesh, read back as an array
        _case("preview", "view", "uniform", 2_000, -1, 256, 256),
        # flying through a mid-size scene: camera inside, image stays on the GPU
        _case("fly_through", "view_device", "gmm", 30_000, 2, 1280, 720, inside=True),
        # rendering a set of held-out views of one size
        _case("render_set", "views", "gmm", 30_000, 1, 800, 800, views=8),
        # fitting with torch autograd, the plain small configuration (base colours)
        _case("autograd_small", "autograd", "uniform", 2_000, -1, 512, 512),
        # fitting with torch autograd, SH degree 3 (the gradient-check configuration)
        _case("autograd_sh3", "autograd", "gmm", 10_000, 3, 512, 512),
        # feature channels and geometry maps with their gradients; sizes no tile divides
        _case("aux_features", "aux", "gmm", 10_000, -1, 637, 421, aux=4),
        # per-tet error statistics that drive densification
        _case("error_stats", "error", "uniform", 10_000, 0, 800, 600),
        # reference-style training loop: one view, target in host memory, odd size
        _case("train_one_view", "train", "gmm", 20_000, -1, 801, 603, targets="host"),
        # data-parallel step: gradients of a rank's views, then the shared update
        _case("accumulate_dp", "accumulate", "gmm", 20_000, 3, 512, 512, views=4),
        # the training-loop configuration's step: eight square views, graph replay
        _case("train_800", "train_views", "gmm", 30_000, 3, 800, 800, views=8),
        # the batched configuration: sixteen views of mixed resolution
        _case("train_mixed16", "train_views", "gmm", 100_000, 3, 0, 0, views=16),
        # large regular mesh at full HD: many small tets
        _case("train_hd_grid", "train_views", "grid", 56, 3, 1920, 1080, views=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(("view", "view_device", "views", "autograd", "aux", "error", "train", "accumulate",
                       "train_views", "train_views"))
    cloud = rng.choice(("uniform", "gmm", "gmm", "grid"))
    points = rng.randint(3, 40) if cloud == "grid" else _log(rng, 300, 40_000)
    many = path in ("views", "accumulate", "train_views")
    width, height = _log(rng, 48, 1400), _log(rng, 48, 1100)
    views = rng.randint(1, max(1, min(12, 6_000_000 // (width * height)))) if many else 1
    if many and rng.random() < 0.25:
        width = height = 0
        views = rng.randint(2, 10)
    return dict(path=path, cloud=cloud, points=points, sh=rng.choice((-1, 0, 1, 2, 3, 3)), width=width, height=height,
                views=views, inside=path in ("view", "view_device") and rng.random() < 0.3,
                aux=rng.randint(1, 8) if path == "aux" else 0,
                targets="host" if path == "train" else rng.choice(("host", "device")))


# ----------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=32)
def _topology(cloud, points):
    """(float64 points in about [-1, 1]^3, int64 tets [M, 4])."""
    rng = np.random.default_rng(points)
    if cloud == "grid":
        n = points + 1
        z, y, x = np.meshgrid(np.arange(n), np.arange(n), np.arange(n), indexing="ij")
        p = np.stack([x, y, z], -1).reshape(-1, 3) * (2.0 / points) - 1.0
        p = p + (rng.random(p.shape) - 0.5) * (0.2 / points)
        z, y, x = (a.reshape(-1) for a in np.meshgrid(*[np.arange(points)] * 3, indexing="ij"))
        c = [(x + i) + (y + j) * n + (z + k) * n * n for k in (0, 1) for j in (0, 1) for i in (0, 1)]
        tets = np.stack([np.stack([c[i] for i in q], -1) for q in
                         ((0, 1, 3, 5), (0, 3, 2, 6), (0, 4, 5, 6), (3, 5, 6, 7), (0, 3, 5, 6))], 1)
        return p, tets.reshape(-1, 4).astype(np.int64)
    p = uniform_cloud(points, rng) if cloud == "uniform" else gmm_cloud(points, rng)
    return p, delaunay_tets(p).reshape(-1, 4).astype(np.int64)


def _circumdata(v, tets):
    """(centre, squared radius) per tet, float32 [M, 4], from float32 vertices."""
    p = v.double()[tets]
    a, b, c = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0], p[:, 3] - p[:, 0]
    bc, ca, ab = (torch.linalg.cross(i, j) for i, j in ((b, c), (c, a), (a, b)))
    den = 2.0 * (a * bc).sum(1, keepdim=True)
    den = torch.where(den.abs() < 1e-12, torch.ones_like(den), den)
    r = ((a * a).sum(1, keepdim=True) * bc + (b * b).sum(1, keepdim=True) * ca + (c * c).sum(1, keepdim=True) * ab) / den
    return torch.cat([p[:, 0] + r, (r * r).sum(1, keepdim=True)], 1).float()


def _inputs(case, seed):
    """Seeded mesh and parameters (float32 CUDA tensors), cameras and targets."""
    rng = np.random.default_rng([seed, 17])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) + 1)

    def randn(*s):
        return torch.randn(*s, generator=gen, device="cuda")

    def rand(*s):
        return torch.rand(*s, generator=gen, device="cuda")

    p, tets = _topology(case["cloud"], case["points"])
    q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    if np.linalg.det(q) < 0:
        q[:, 0] = -q[:, 0]
    d = {"tets": torch.from_numpy(tets).cuda(), "vertices": torch.from_numpy((p @ q).astype(np.float32)).cuda()}
    m, sh = tets.shape[0], case["sh"]
    d["densities"] = torch.exp(randn(m))
    d["color_grads"] = 0.1 * randn(m, 3)
    d["circumdata"] = _circumdata(d["vertices"], d["tets"])
    if sh >= 0:
        d["sh_coeffs"] = 0.5 * randn(m, 3, (sh + 1) ** 2)
        d["base_colors"] = 0.5 + 0.28209479177387814 * d["sh_coeffs"][:, :, 0].contiguous()
    else:
        d["base_colors"] = 0.5 + 0.14 * randn(m, 3)
    w, h = case["width"], case["height"]
    if case["inside"]:
        at = rng.uniform(-0.3, 0.3, size=3)
        to = at + np.array([math.cos(seed), math.sin(seed), rng.uniform(-0.3, 0.3)])
        cams = [make_camera(tuple(at), tuple(to), 70.0, w, h)]
    else:
        cams = orbit_cameras(case["views"], seed=int(rng.integers(1 << 30)), radius=(2.5, 4.0),
                             resolutions=MIXED if w == 0 else ((w, h),))
    d["cams"] = cams
    n_pix = sum(c.width * c.height for c in cams)
    if case["path"] in ("autograd", "train", "accumulate", "train_views"):
        d["gt"] = rand(3 * n_pix)
    if case["path"] == "aux":
        d["aux_data"] = rand(m, case["aux"])
        d["dl"] = randn(n_pix, 4) / n_pix
        d["dl_aux"] = randn(n_pix, case["aux"]) / n_pix
    if case["path"] == "error":
        d["pixel_err"], d["ssim_err"] = rand(n_pix), rand(n_pix)
    return d


def _host(x):
    return x.reshape(-1).cpu().numpy()


def prepare(case, seed):
    d = _inputs(case, seed)
    cams = d["cams"]
    idx = np.ascontiguousarray(_host(d["tets"]).astype(np.uint32))
    args = (_host(d["vertices"]), idx, _host(d["base_colors"]), _host(d["densities"]), _host(d["color_grads"]),
            _host(d["circumdata"]))
    sh = dict(sh_coeffs=_host(d["sh_coeffs"]), sh_degree=case["sh"]) if case["sh"] >= 0 else {}
    s = {"case": case, "cams": cams}
    if case["path"] == "autograd":
        s["module"] = RMeshModule(*args, cams[0].width, cams[0].height, device="cuda", **sh)
        s["gt"] = d["gt"].view(cams[0].height, cams[0].width, 3)
        return s
    s["r"] = r = RMeshRenderer(*args, cams[0].width, cams[0].height, case["aux"], **sh)
    n_pix = sum(c.width * c.height for c in cams)
    if case["path"] in ("view_device", "views"):
        s["out"] = torch.empty(4 * n_pix, dtype=torch.float32, device="cuda")
    if "gt" in d:
        s["gt"] = _host(d["gt"]) if case["targets"] == "host" else d["gt"]
    if case["path"] == "aux":
        r.set_aux_data(_host(d["aux_data"]))
        s["dl"], s["dl_aux"] = _host(d["dl"]), _host(d["dl_aux"])
    if case["path"] == "error":
        s["pixel_err"], s["ssim_err"] = _host(d["pixel_err"]), _host(d["ssim_err"])
    return s


# ------------------------------------------------------------------- run
def _slots(r):
    """The renderer's gradient buffer; its memory lives as long as the renderer,
    which the returned tensor keeps."""
    g = r.grad_slots()
    g.owner = r
    return g


def run(s):
    path, c = s["case"]["path"], s["cams"][0]
    cam = (c.cam_pos, c.vp, c.c2w_intrinsics)
    if path == "autograd":
        mod = s["module"]
        img = mod(*cam)
        loss = ((img[..., :3] - s["gt"]) ** 2).sum() / (c.width * c.height)
        params = [mod.vertices, mod.densities, mod.color_grads, mod.sh_coeffs if mod.sh_coeffs is not None
                  else mod.base_colors]
        dv, dd, dg, dc = torch.autograd.grad(loss, params)
        return {"image": img.detach(), "d_vertices": dv, "d_densities": dd, "d_color_grads": dg, "d_color": dc}
    r = s["r"]
    if path == "view":
        return {"image": r.forward_tiled(*cam)}
    if path == "view_device":
        return {"image": r.forward_tiled_into(*cam, s["out"])}
    if path == "views":
        return {"image": r.forward_views(s["cams"], out=s["out"])}
    if path == "aux":
        img, aux = r.forward_tiled(*cam, render_aux=True)
        g = r.backward(s["dl"], s["dl_aux"])
        out = {"image": img, "aux": aux}
        out.update((k, v) for k, v in g.items() if k != ("d_base_colors" if s["case"]["sh"] >= 0 else ""))
        return out
    if path == "error":
        img = r.forward_tiled(*cam)
        err, cnt = r.forward_error(s["pixel_err"], s["ssim_err"])
        return {"image": img, "tet_err": err, "tet_count": cnt}
    if path == "train":
        loss = r.train_step(*cam, s["gt"], **LR, loss_type=1, lr_sh=LR_SH)
        return {"loss": [loss], "grads": _slots(r)}
    if path == "accumulate":
        loss = r.accumulate_views(s["cams"], s["gt"], mode="batched")
        r.apply_adam(**LR, lr_sh=LR_SH)
        return {"loss": loss, "grads": _slots(r)}
    loss = r.train_step_views(s["cams"], s["gt"], **LR, lr_sh=LR_SH, mode="graph")
    return {"loss": loss, "grads": _slots(r)}


# ------------------------------------------------- what a pass cannot do without
def _sizes(case):
    n = (case["points"] + 1) ** 3 if case["cloud"] == "grid" else case["points"]
    m = 5 * case["points"] ** 3 if case["cloud"] == "grid" else 6.7 * case["points"]
    px = case["views"] * (case["width"] * case["height"] or 0.5 * (256 ** 2 + 1024 ** 2))
    return n, m, px


def work(case):
    """Bytes: parameters and targets read once, images and gradients written
    once.  Operations: the (pixel, tet) crossings on the average ray through the
    mesh (about 2.7 per cube root of the vertex count over the whole image) times
    the arithmetic of one crossing: four plane hits, the segment integral and the
    blend (90), and in a step with gradients their adjoint (250 more)."""
    n, m, px = _sizes(case)
    nc = (case["sh"] + 1) ** 2 if case["sh"] >= 0 else 1
    params = 12 * n + m * (16 + 16 + 4 + 12 + 12 * nc)
    grad = case["path"] not in ("view", "view_device", "views", "error")
    hits = 2.7 * n ** (1 / 3) * px
    out = {"aux": 16 + 4 * (8 + case["aux"]) + 4 * (4 + case["aux"]), "error": 16 + 8}.get(case["path"], 16)
    by = params + px * (12 if case["path"] in ("train", "accumulate", "train_views") else out)
    by += m * 72 if case["path"] == "error" else 0
    by += (12 * n + m * (16 + 12 * nc)) if grad else 0
    # Adam: parameters written, moments read and written
    by += 5 * (12 * n + m * (16 + (12 * nc if case["sh"] >= 0 else 0))) if case["path"] in ("train", "accumulate",
                                                                                        "train_views") else 0
    return {"bytes": float(by), "flops": float(hits * (340 if grad else 90))}


def tolerance(case):
    """Images differ from the same in 64 bits by 1e-6 to 1.5e-5 (thin tets, whose
    crossing is a difference of two near-equal distances), single pixels by up to
    1.6e-2.  The gradients of such tets' vertices cancel further: 1e-4 to 6e-3 on
    the Delaunay meshes and 1.5e-2 on the regular one, single values by more than
    themselves.  Repeated runs (sums in another order) agree to 1e-6."""
    if case["path"] in ("view", "view_device", "views", "error"):
        return {"rel": 6e-5, "max": 0.06, "differ": 1e-3}
    return {"rel": 1e-2, "max": 0.9, "differ": 1e-3}


# ------------------------------------------------------- the same in 64 bits
_FACES = ((0, 2, 1, 3), (1, 2, 3, 0), (0, 3, 2, 1), (3, 0, 1, 2))
_SPAN = 3_000_000  # crossings taken through autograd at a time


def _sh_color(q, corners, g, cam):
    """softplus(SH(direction to the centroid) + 0.5 + g.(v0 - centroid)), beta 10."""
    cen = corners.mean(1)
    d = cen - cam
    d = d / d.norm(dim=1, keepdim=True)
    x, y, z = d.unbind(1)
    b = [torch.full_like(x, 0.28209479177387814)]
    if q.shape[2] > 1:
        k = 0.4886025119029199
        b += [-k * y, k * z, -k * x]
    if q.shape[2] > 4:
        b += [1.0925484305920792 * x * y, -1.0925484305920792 * y * z, 0.31539156525252005 * (2 * z * z - x * x - y * y),
              -1.0925484305920792 * x * z, 0.5462742152960396 * (x * x - y * y)]
    if q.shape[2] > 9:
        b += [-0.5900435899266435 * y * (3 * x * x - y * y), 2.890611442640554 * x * y * z,
              -0.4570457994644658 * y * (4 * z * z - x * x - y * y),
              0.3731763325901154 * z * (2 * z * z - 3 * x * x - 3 * y * y),
              -0.4570457994644658 * x * (4 * z * z - x * x - y * y), 1.445305721320277 * z * (x * x - y * y),
              -0.5900435899266435 * x * (x * x - 3 * y * y)]
    v = (q * torch.stack(b, 1)[:, None, :]).sum(2) + 0.5 + (g * (corners[:, 0] - cen)).sum(1, keepdim=True)
    return torch.nn.functional.softplus(v, beta=10.0, threshold=20.0)


def _cuda64(x):
    return torch.as_tensor(np.asarray(x), dtype=torch.float64, device="cuda")


def _rays(c):
    """Unit ray directions [H, W, 3]."""
    k = _cuda64(c.c2w_intrinsics)
    y, x = torch.meshgrid(torch.arange(c.height, device="cuda", dtype=torch.float64) + 0.5,
                          torch.arange(c.width, device="cuda", dtype=torch.float64) + 0.5, indexing="ij")
    u = torch.stack([(x - k[14]) / k[12], (y - k[15]) / k[13], torch.ones_like(x)], -1)
    u = u / u.norm(dim=-1, keepdim=True)
    w = u @ torch.stack([k[0:3], k[4:7], k[8:11]])
    return w / w.norm(dim=-1, keepdim=True)


def _planes(corners, cam):
    """Inward normals [M, 4, 3] and n.(a - cam) [M, 4]."""
    n, num = [], []
    for a, b, c, o in _FACES:
        va = corners[:, a]
        q = torch.linalg.cross(corners[:, c] - va, corners[:, b] - va)
        s = torch.where((q * (corners[:, o] - va)).sum(1, keepdim=True) < 0, -1.0, 1.0)
        q = q * s
        n.append(q)
        num.append((q * (va - cam)).sum(1))
    return torch.stack(n, 1), torch.stack(num, 1)


def _segments(normals, nums, dirs):
    """Entry and exit distance of rays with their tets and the entry face."""
    den = (normals * dirs[:, None, :]).sum(2)
    t = nums / torch.where(den == 0, torch.ones_like(den), den)
    t0, face = torch.where(den > 0, t, torch.full_like(t, -3e38)).max(1)
    t1 = torch.where(den < 0, t, torch.full_like(t, 3e38)).min(1)[0]
    return t0, t1, face


def _crossings(c, corners32, dens32, circ32):
    """(tet, pixel) of every crossing, grouped by pixel and near to far inside
    it, over the tets that the renderer keeps (its culls and its depth order are
    defined on float32 values), in runs of whole rows."""
    cam = _cuda64(c.cam_pos)
    corners = corners32.double()
    vp = _cuda64(c.vp).view(4, 4).t()
    h = torch.cat([corners, torch.ones_like(corners[..., :1])], 2) @ vp.t()
    keep = (h[..., 3] > 0).all(1)
    ndc = h[..., :3] / (h[..., 3:] + 1e-6)
    lo, hi = ndc.amin(1), ndc.amax(1)
    keep &= (hi[:, 0] >= -1) & (lo[:, 0] <= 1) & (hi[:, 1] >= -1) & (lo[:, 1] <= 1) & (lo[:, 2] <= 1)
    ext = (hi - lo)[:, :2] * torch.tensor([c.width, c.height], device="cuda")
    keep &= ext.prod(1) >= 1.0
    longest = (corners[:, :, None] - corners[:, None]).square().sum(3).amax((1, 2)).sqrt()
    keep &= dens32.double() * longest >= 0.01
    at = torch.as_tensor(c.cam_pos, device="cuda")
    e = [circ32[:, i] - at[i] for i in range(3)]
    depth = (e[0] * e[0] + e[1] * e[1]) + e[2] * e[2] - circ32[:, 3]
    key = depth.view(torch.int32).long()  # ~bits, unsigned and ascending, is back to front
    key = (~key) & 0xFFFFFFFF
    ids = torch.nonzero(keep).squeeze(1)
    # the renderer's lists are ascending (ties by tet id) and walked from their end
    ids = ids[torch.sort(key[ids], stable=True)[1]].flip(0)
    clip = h[ids]
    px = (clip[..., 0] / clip[..., 3] + 1) * 0.5 * c.width
    py = (1 - clip[..., 1] / clip[..., 3]) * 0.5 * c.height
    x0 = (px.amin(1) - 0.51).ceil().clamp(0, c.width - 1).long()
    x1 = (px.amax(1) - 0.49).floor().clamp(-1, c.width - 1).long()
    y0 = (py.amin(1) - 0.51).ceil().clamp(0, c.height - 1).long()
    y1 = (py.amax(1) - 0.49).floor().clamp(-1, c.height - 1).long()
    ok = (x1 >= x0) & (y1 >= y0)
    ids, x0, x1, y0, y1 = (v[ok] for v in (ids, x0, x1, y0, y1))
    normals, nums = _planes(corners, cam)
    dirs = _rays(c)
    per_row = torch.zeros(c.height + 1, dtype=torch.float64, device="cuda")
    per_row.index_add_(0, y0, (x1 - x0 + 1).double())
    per_row.index_add_(0, y1 + 1, -(x1 - x0 + 1).double())
    per_row = per_row.cumsum(0)[:-1].cpu().numpy()
    r0 = 0
    while r0 < c.height:
        r1, total = r0, 0.0
        while r1 < c.height and (r1 == r0 or total + per_row[r1] <= 4 * _SPAN):
            total += per_row[r1]
            r1 += 1
        sel = torch.nonzero((y1 >= r0) & (y0 < r1)).squeeze(1)
        if sel.numel():
            a, b = y0[sel].clamp(min=r0), y1[sel].clamp(max=r1 - 1)
            w = x1[sel] - x0[sel] + 1
            n = w * (b - a + 1)
            own = torch.repeat_interleave(torch.arange(sel.numel(), device="cuda"), n)
            k = torch.arange(own.numel(), device="cuda") - (n.cumsum(0) - n)[own]
            pix = (a[own] + k // w[own]) * c.width + x0[sel][own] + k % w[own]
            tet = ids[sel][own]
            hit = []
            for i in range(0, own.numel(), _SPAN):
                t = tet[i:i + _SPAN]
                t0, t1, _ = _segments(normals[t], nums[t], dirs.view(-1, 3)[pix[i:i + _SPAN]])
                hit.append(t0 < t1)
            hit = torch.cat(hit)
            pix, tet = pix[hit], tet[hit]
            pix, order = torch.sort(pix, stable=True)
            yield r0, r1, tet[order], pix
        else:
            yield r0, r1, ids[:0], ids[:0]
        r0 = r1


def _composite(c, cam, tet, pix, corners, dens, color, g, dirs):
    """Per crossing: colour, optical depth, transmittance before it, t0, t1, face."""
    normals, nums = _planes(corners, cam)
    d = dirs.view(-1, 3)[pix]
    t0, t1, face = _segments(normals[tet], nums[tet], d)
    base = (color + (g * (cam - corners[:, 0])).sum(1, keepdim=True))[tet]
    slope = (g[tet] * d).sum(1, keepdim=True)
    c0, c1 = (base + slope * t0[:, None]).clamp(min=0), (base + slope * t1[:, None]).clamp(min=0)
    od = (dens[tet] * (t1 - t0)).clamp(1e-8, 88.0)
    al = torch.exp(-od)
    ph = torch.where(od < 1e-4, 1 - od * (0.5 - od * (1 / 6 - od / 24)), -torch.expm1(-od) / od)
    col = c1 * (ph - al)[:, None] + c0 * (1 - ph)[:, None]
    first = torch.ones_like(pix, dtype=torch.bool)
    first[1:] = pix[1:] != pix[:-1]
    run_ = torch.cumsum(od, 0) - od
    start = run_[torch.nonzero(first).squeeze(1)][torch.cumsum(first.long(), 0) - 1] if pix.numel() else run_
    T = torch.exp(start - run_)
    return col, od, T, t0, t1, face, al, ph, normals, d


def exact(case, seed):
    d = _inputs(case, seed)
    path, cams = case["path"], d["cams"]
    tets = d["tets"]
    grad = path not in ("view", "view_device", "views", "error")
    corners32 = d["vertices"][tets]
    corners = corners32.double().requires_grad_(grad)
    dens = d["densities"].double().requires_grad_(grad)
    g = d["color_grads"].double().requires_grad_(grad)
    leaves = [corners, dens, g]
    if case["sh"] >= 0:
        col_p = d["sh_coeffs"].half().double().requires_grad_(grad)  # the coefficients are read as 16-bit values
    else:
        col_p = d["base_colors"].double().requires_grad_(grad)
    leaves.append(col_p)
    aux_p = d["aux_data"].double().requires_grad_(True) if path == "aux" else None
    if aux_p is not None:
        leaves.append(aux_p)
    images, auxs, losses, at = [], [], [], 0
    m = tets.shape[0]
    stats = torch.zeros(m, 16, dtype=torch.float64, device="cuda") if path == "error" else None
    for c in cams:
        n_pix, cam, dirs = c.width * c.height, _cuda64(c.cam_pos), _rays(c)
        image = torch.zeros(n_pix, 4, dtype=torch.float64, device="cuda")
        aux_img = torch.zeros(n_pix, 8 + case["aux"], dtype=torch.float64, device="cuda") if path == "aux" else None
        gt = d["gt"][3 * at:3 * (at + n_pix)].double().view(-1, 3) if "gt" in d else None
        loss = 0.0
        for r0, r1, tet, pix in _crossings(c, corners32, d["densities"], d["circumdata"]):
            rows = slice(r0 * c.width, r1 * c.width)
            with torch.set_grad_enabled(grad):
                color = _sh_color(col_p, corners, g, cam) if case["sh"] >= 0 else col_p
                col, od, T, t0, t1, face, al, ph, normals, dd = _composite(c, cam, tet, pix, corners, dens, color, g, dirs)
                see = T >= 1e-6
                Ts, ods = T * see, od * see
                loc = pix - r0 * c.width
                z = torch.zeros(rows.stop - rows.start, dtype=torch.float64, device="cuda")
                rgb = z[:, None].repeat(1, 3).index_add(0, loc, col * Ts[:, None])
                A = 1 - torch.exp(-z.index_add(0, loc, ods))
                out = torch.cat([rgb, A[:, None]], 1)
                total = None
                if gt is not None:
                    total = (rgb - gt[rows]).square().sum() / n_pix
                    loss += float(total.detach())
                if path == "aux":
                    wt = (1 - al) * Ts
                    custom = torch.zeros(z.numel(), case["aux"], dtype=torch.float64, device="cuda").index_add(
                        0, loc, wt[:, None] * aux_p[tet])
                    total = (out * d["dl"].double()[rows]).sum() + (custom * d["dl_aux"].double()[rows]).sum()
                if total is not None:
                    total.backward()
            image[rows] = out.detach()
            if path == "aux":
                with torch.no_grad():
                    nrm = normals[tet, face]
                    nrm = -nrm / nrm.norm(dim=1, keepdim=True)
                    mid = 0.5 * (t0 + t1)
                    wc = wt * mid
                    xlx = lambda v: torch.where(v > 1e-20, v * torch.log(v.clamp(min=1e-300)), torch.zeros_like(v))  # noqa: E731
                    cols = torch.cat([wt[:, None] * nrm, (Ts * ((ph - al) * t1 + (1 - ph) * t0))[:, None], wt[:, None],
                                      xlx(wt)[:, None], wc[:, None], xlx(wc)[:, None]], 1)
                    aux_img[rows, :8] = torch.zeros(z.numel(), 8, dtype=torch.float64, device="cuda").index_add(0, loc, cols)
                    aux_img[rows, 8:] = custom.detach()
            if path == "error":
                w = (T * od) * (torch.log(T) >= -5.5)
                pe, se = d["pixel_err"].double()[pix], d["ssim_err"].double()[pix]
                cen = corners.mean(1)[tet]
                zero = torch.zeros_like(w)
                stats.index_add_(0, tet, torch.stack(
                    [w, w * pe, w * pe * pe, zero, zero, w * se] + [w * (cam[i] + dd[:, i] * t0) for i in range(3)] +
                    [w * (cam[i] + dd[:, i] * t1) for i in range(3)] + [w] + [w * cen[:, i] for i in range(3)], 1))
            del color, col, od, T, t0, t1, face, al, ph, normals, dd
        images.append(image)
        losses.append(loss)
        if path == "aux":
            auxs.append(aux_img.view(c.height, c.width, -1))
        at += n_pix
    image = torch.cat(images)
    c = cams[0]
    if path == "views":
        return {"image": image.view(-1)}
    if path == "view_device":
        return {"image": image.view(-1)}
    image = image.view(c.height, c.width, 4) if len(cams) == 1 else None
    if path == "view":
        return {"image": image}
    if path == "error":
        return {"image": image, "tet_err": stats, "tet_count": None}
    dv = torch.zeros(d["vertices"].shape, dtype=torch.float64, device="cuda").index_add(
        0, tets.reshape(-1), corners.grad.reshape(-1, 3))
    if path == "autograd":
        return {"image": image, "d_vertices": dv.view(-1), "d_densities": dens.grad, "d_color_grads": g.grad.view(-1),
                "d_color": col_p.grad.reshape(-1)}
    if path == "aux":
        return {"image": image, "aux": auxs[0], "d_vertices": dv.view(-1), "d_densities": dens.grad,
                "d_color_grads": g.grad.view(-1), ("d_sh_coeffs" if case["sh"] >= 0 else "d_base_colors"): col_p.grad.reshape(-1),
                "d_aux_data": aux_p.grad.view(-1)}
    z3 = torch.zeros(m, 3, dtype=torch.float64, device="cuda")
    slots = torch.cat([dens.grad[:, None], z3 if case["sh"] >= 0 else col_p.grad, g.grad, corners.grad.view(m, 12),
                       z3[:, :1]], 1).reshape(-1)
    if case["sh"] >= 0:
        slots = torch.cat([slots, col_p.grad.reshape(-1)])
    return {"loss": losses if path == "train" else _cuda64(losses), "grads": slots}
