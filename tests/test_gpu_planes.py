"""The branch-free ray-plane arithmetic (needs a B200): its quotient and its choice of
faces against the general path, value by value, and meshes scaled past both ends of the
range in which it is used against the CPU oracle."""
from __future__ import annotations

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT, make_renderer, rel_l2

pytestmark = pytest.mark.gpu

PROBE = r'''
#include "tile.cuh"
using namespace rm;
__device__ uint32_t mix(uint32_t x) {
  x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; return x ^ (x >> 16);
}
// a number of either sign, its exponent uniform in [lo, hi], its significand random or,
// one time in four, all ones or all zeros but the last bits
__device__ float number(uint32_t& s, int lo, int hi) {
  const uint32_t a = mix(s += 0x9e3779b9u), b = mix(s += 0x9e3779b9u);
  uint32_t m = a & 0x7fffffu;
  if ((b & 3u) == 0u) m = (b & 4u) ? 0x7fffffu - (m & 7u) : (m & 7u);
  const uint32_t e = (uint32_t)(127 + lo) + (b >> 8) % (uint32_t)(hi - lo + 1);
  return __uint_as_float((b & 8u) << 28 | e << 23 | m);
}
__global__ void quotients(uint32_t seed, int per, unsigned long long* wrong) {
  uint32_t s = mix(seed ^ (blockIdx.x * blockDim.x + threadIdx.x + 1u));
  unsigned long long bad = 0;
  for (int i = 0; i < per; ++i) {
    const float den = number(s, -66, 59), num = (i & 255) ? number(s, -60, 59) : 0.0f;
    if (fabsf(den) < 1e-20f) continue;
    bad += __float_as_uint(plain_quotient(num, den)) != __float_as_uint(__fdiv_rn(num, den));
  }
  if (bad) atomicAdd(wrong, bad);
}
__global__ void faces(uint32_t seed, int per, unsigned long long* wrong, unsigned long long* taken) {
  uint32_t s = mix(seed ^ (blockIdx.x * blockDim.x + threadIdx.x + 1u));
  unsigned long long bad = 0, n = 0;
  for (int i = 0; i < per; ++i) {
    float4 p[4];
    // equal planes now and then: ties of t
    for (int f = 0; f < 4; ++f) {
      p[f] = make_float4(number(s, -6, 3), number(s, -6, 3), number(s, -6, 3), number(s, -6, 3));
      if (f && (mix(s += 1u) & 7u) == 0u) p[f] = p[f - 1];
    }
    const float dx = number(s, -4, 0), dy = number(s, -4, 0), dz = number(s, -4, 0);
    float a0, a1, b0, b1, c0, c1;
    int am, ax, bm, bx, cm, cx;
    bool plain, plain2;
    const bool h = intersect4_plain<true>(p, dx, dy, dz, a0, a1, am, ax, plain);
    const bool h2 = intersect4_plain<false>(p, dx, dy, dz, c0, c1, cm, cx, plain2);
    const bool g = intersect4(p, nullptr, dx, dy, dz, b0, b1, bm, bx);
    if (!plain) continue;
    ++n;
    bad += h != g || h2 != g || !plain2 || a0 != b0 || a1 != b1 || c0 != b0 || c1 != b1 || am != bm || ax != bx;
  }
  if (bad) atomicAdd(wrong, bad);
  atomicAdd(taken, n);
}
extern "C" int run(unsigned long long* out) {
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, 24) != cudaSuccess) return 1;
  cudaMemset(d, 0, 24);
  quotients<<<592, 256>>>(1u, 2000, d);
  faces<<<592, 256>>>(2u, 200, d + 1, d + 2);
  const cudaError_t e = cudaMemcpy(out, d, 24, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e != cudaSuccess || cudaGetLastError() != cudaSuccess;
}
'''


def test_quotient_and_faces_equal_the_general_path(tmp_path):
    """3.0e8 quotients against __fdiv_rn and 3e7 rays against intersect4, bit for bit."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    from rmesh_b200 import build

    src, so = tmp_path / "probe.cu", tmp_path / "probe.so"
    src.write_text(PROBE)
    subprocess.run([nvcc, *build.NVCC_FLAGS, "-Xcompiler", "-fvisibility=default", "-I",
                    os.path.join(ROOT, "rmesh_b200", "csrc"), str(src), "-o", str(so)], check=True)
    out = (ctypes.c_ulonglong * 3)()
    assert ctypes.CDLL(str(so)).run(out) == 0
    assert out[0] == 0 and out[1] == 0
    assert out[2] > 10_000_000


# powers of two: n.(a - cam) leaves [2^-60, 2^60] for some tets from 2^20 and 2^-18 on, for
# all at 2^24 and 2^-23; normals exceed 2^58 at 2^31
@pytest.mark.parametrize("e", [19, 20, 21, 24, 31, -18, -19, -20, -23])
def test_meshes_beyond_the_branch_free_range(c1_scene, oracle32, e):
    from rmesh_b200.camera import make_camera

    k = 2.0 ** e
    sc = dict(c1_scene)
    sc["vertices"] = (c1_scene["vertices"] * k).astype(np.float32)
    sc["densities"] = (c1_scene["densities"] / k).astype(np.float32)
    sc["color_grads"] = (c1_scene["color_grads"] / k).astype(np.float32)
    c = c1_scene["circumdata"].reshape(-1, 4).astype(np.float64)
    sc["circumdata"] = np.concatenate([c[:, :3] * k, c[:, 3:] * k * k], 1).astype(np.float32).ravel()
    cam = make_camera((1.9 * k, -2.1 * k, 1.1 * k), (0.0, 0.0, 0.0), 55.0, 150, 110, near=0.01 * k, far=100.0 * k)
    r = make_renderer(sc, cam)
    img = r.forward_tiled(cam.cam_pos, cam.vp, cam.c2w_intrinsics)
    ref = oracle32.forward_tiled(sc, cam)
    assert ref["P"] > 1000
    tiles, tets = r.debug_pairs()
    np.testing.assert_array_equal(tiles, ref["key_hi"])
    np.testing.assert_array_equal(tets, ref["vals"])
    assert np.abs(img - ref["image"]).max() <= 1e-4
    gt = np.random.default_rng(2).uniform(0, 1, (cam.height, cam.width, 3)).astype(np.float32)
    _, dl = oracle32.loss(ref["image"], gt, 1)
    g = r.backward(dl)
    go = oracle32.backward(sc, cam, dl, ref)
    for q in go:
        assert rel_l2(g[q], go[q]) <= 1e-3, q
    r.close()
