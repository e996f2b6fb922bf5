"""The receivers' footprint layout against the atlases it is derived from: atlases
uploaded in parts, then gathered at the tiles' and cages' edges (axis directions of
either sign of zero, directions on the octahedral seams, positions on probes, on the
box and outside it, ragged counts), compared with a bilinear, trilinear read of the
uploaded RGBA16F texels in 64 bits (the receiver gather's bar, 1e-3 relative). A
zero normal gives 0, as before."""
import ctypes as C

import numpy as np
import pytest
import torch

from speedball_b200 import _abi, synth

import gpu_util as gu

pytestmark = pytest.mark.gpu


def _oct(n):
    s = np.abs(n).sum(1, keepdims=True)
    n = n / np.maximum(s, 1e-20)
    f = (1 - np.abs(n[:, [1, 0]])) * np.where(n[:, :2] >= 0, 1.0, -1.0)
    return np.where(n[:, 2:] < 0, f, n[:, :2]) * 0.5 + 0.5


def _expected(atlas, res, lo, size, pos, nrm):
    res, lo, size = np.array(res), np.array(lo), np.array(size)
    gf = (pos - lo) / (size / np.maximum(res - 1, 1))
    base = np.clip(np.floor(gf), 0, np.maximum(res - 2, 0))
    frac = np.clip(gf - base, 0, 1)
    uv = 0.5 + _oct(nrm) * 6
    x0, y0 = np.floor(uv).astype(int).T
    fx, fy = (uv - np.floor(uv)).T[:, :, None]
    acc, ws = 0.0, 0.0
    for i in range(8):
        d = np.array([i & 1, i >> 1 & 1, i >> 2 & 1])
        p = (base + d).astype(int)
        w = np.prod(np.where(d > 0, frac, 1 - frac), 1) + 1e-4
        ty, tx = (p[:, 2] * res[1] + p[:, 1]) * 8 + y0, p[:, 0] * 8 + x0
        e = (atlas[ty, tx] * (1 - fx) + atlas[ty, tx + 1] * fx) * (1 - fy) + \
            (atlas[ty + 1, tx] * (1 - fx) + atlas[ty + 1, tx + 1] * fx) * fy
        acc = acc + e[:, :3] * w[:, None]
        ws = ws + w
    return acc / ws[:, None]


@pytest.mark.parametrize("res", [(2, 2, 2), (3, 5, 2), (7, 4, 6)])
def test_gather_reads_the_uploaded_texels(res):
    scene = synth.room_spheres(1)
    scene.meta["grid"] = dict(scene.meta["grid"], res=res)
    f = gu.make_field(scene)
    try:
        lo, size = scene.meta["grid"]["gridMin"], scene.meta["grid"]["gridSize"]
        rng = np.random.default_rng(sum(res))
        W, H = res[0] * 8, res[1] * res[2] * 8
        atlas = rng.uniform(0.1, 4.0, (H, W, 4)).astype(np.float16)
        flat, cut = atlas.reshape(-1), (W * 4 * 5) + 12  # a part that ends inside a row
        for a, b in ((0, cut), (cut, flat.size)):
            part = np.ascontiguousarray(flat[a:b])
            _abi.check(f._lib.sb_upload_range(f.ctx, _abi.BUF["IRRADIANCE_ATLAS"], a, b - a, _abi.ptr(part)), f.ctx)
        dirs = [s * np.eye(3)[a] for a in range(3) for s in (1, -1)]
        dirs += [np.array(v, float) for v in ((1, 1, 0), (-1, 1, 0), (0.0, 1, -1), (-0.0, 1, -1), (1, -0.0, -2),
                                              (3, 4, -5), (1e-3, -1e-3, -1), (200, 300, 100))]
        cell = np.array(size) / (np.array(res) - 1)
        pts = [np.array(lo), np.array(lo) + size, np.array(lo) + cell, np.array(lo) - 1.0, np.array(lo) + 1.5 * np.array(size),
               np.array(lo) + 0.5 * cell]
        pts += [np.array(lo) + np.array(size) * rng.random(3) for _ in range(9)]
        pos = np.array([p for p in pts for _ in dirs])
        nrm = np.array([d for _ in pts for d in dirs])
        prm = _abi.sb_gather_params()
        f._lib.sb_gather_params_defaults(C.byref(prm))
        prm.normalBias[0] = 0.0
        for n in (1, 33, pos.shape[0]):
            p4, n4 = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
            p4[:, :3], n4[:, :3] = pos[:n], nrm[:n]
            n4[0, :3] = 0.0
            dev = [torch.from_numpy(a).cuda() for a in (p4, n4)] + [torch.zeros(n, 4, device="cuda")]
            torch.cuda.synchronize()
            ptr = [C.c_void_p(t.data_ptr()) for t in dev]
            _abi.check(f._lib.sb_gather_irradiance(f.ctx, C.byref(prm), ptr[0], ptr[1], ptr[1], n, ptr[2]), f.ctx)
            f.synchronize()
            got = dev[2].cpu().numpy()
            want = _expected(atlas.astype(np.float64), res, lo, size, p4[1:, :3].astype(np.float64),
                             n4[1:, :3].astype(np.float64))
            assert np.array_equal(got[0], np.array([0, 0, 0, 1], np.float32))
            assert np.all(np.abs(got[1:, :3] - want) <= 1e-3 * np.abs(want))
    finally:
        f.dispose()
