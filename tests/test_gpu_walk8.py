"""The warp walks of the 8-wide scene BVH at small and ragged ray counts (part of a
warp, one warp, several, more than one refill), with and without moved slots:
closest hits and occlusion equal those of the binary tree's and the two-level
walk's, which test one ray per lane. Where two triangles are hit at nearly the
same t the walks may name either (the suite's near-tie bar, 1e-6 relative)."""
import ctypes as C

import numpy as np
import pytest

from speedball_b200 import _abi, synth

import gpu_util as gu

pytestmark = pytest.mark.gpu


def _queries(f, ro, rd, dist):
    n = ro.shape[0]
    t, tri, inst = np.zeros(n, np.float32), np.zeros(n, np.int32), np.zeros(n, np.int32)
    _abi.check(f._lib.sb_raycast(f.ctx, _abi.ptr(ro), _abi.ptr(rd), n, _abi.ptr(t), _abi.ptr(tri), _abi.ptr(inst)), f.ctx)
    occ = np.zeros(n, np.uint8)
    _abi.check(f._lib.sb_occluded(f.ctx, _abi.ptr(ro), _abi.ptr(rd), _abi.ptr(dist), n, _abi.ptr(occ)), f.ctx)
    return t, tri, inst, occ


def _kind(f, kind):
    t = _abi.sb_tuning()
    _abi.check(f._lib.sb_get_tuning(f.ctx, C.byref(t)), f.ctx)
    t.bvhKind = kind
    _abi.check(f._lib.sb_set_tuning(f.ctx, C.byref(t)), f.ctx)


@pytest.mark.parametrize("moved", [False, True])
def test_queries_agree_with_the_other_layouts(moved):
    f = gu.make_field(synth.room_spheres(4))
    try:
        f.tick()
        if moved:  # two spheres leave the tree
            for i in (3, 17):
                f._scene.instances[i].world = f._scene.instances[i].world @ synth.trs((0.4, -0.2, 0.1))
            f.markTransformsDirty([3, 17])
            f.tick()
        f.synchronize()
        for n in (1, 31, 32, 33, 1000, 20011):
            rng = np.random.default_rng(n)
            ro = rng.uniform(0.2, 9.8, (n, 3)).astype(np.float32)
            rd = rng.normal(size=(n, 3)).astype(np.float32)
            rd /= np.linalg.norm(rd, axis=1, keepdims=True)
            rd[::7, 1] = 0.0  # axis-parallel in one axis
            dist = rng.uniform(0.0, 6.0, n).astype(np.float32)
            dist[::5] = 0.0
            got = {}
            for kind in (1, 2, 0):
                _kind(f, kind)
                got[kind] = _queries(f, ro, rd, dist)
            _kind(f, 1)
            t, tri, inst, occ = got[1]
            assert not occ[::5].any()
            for kind in (2, 0):
                t2, tri2, inst2, occ2 = got[kind]
                same = (tri == tri2) & (inst == inst2)
                assert np.array_equal(t[same], t2[same])
                assert np.all(np.abs(t - t2)[~same] <= gu.TIE_REL * np.abs(t2)[~same])
                assert np.array_equal(occ, occ2)
            assert (tri >= 0).mean() > 0.9
    finally:
        f.dispose()


@pytest.mark.parametrize("res,rays", [((2, 2, 2), 32), ((3, 2, 5), 48), ((9, 7, 5), 256)])
def test_solve_matches_the_two_level_walk_with_moved_slots(res, rays):
    """A whole solve after slots moved and one BLAS deformed: irradiance and depth of
    the 8-wide walk's fields equal the two-level walk's up to near-ties (the texel
    bar of the parity tests)."""
    out = []
    for kind in (1, 0):
        scene = synth.atrium(9, total_tris=20_000)
        scene.meta["grid"] = dict(scene.meta["grid"], res=res, rays=rays)
        f = gu.make_field(scene)
        try:
            _kind(f, kind)
            for frame in range(2):
                mats, pos = synth.atrium_motion(scene, frame)
                for i, m in mats.items():
                    scene.instances[i].world = m
                if frame:
                    scene.meshes[scene.meta["deformer"]].positions = pos
                    f.markDeformsDirty()
                f.markTransformsDirty(list(mats))
                f.tick()
            f.synchronize()
            P = f._probeTotal
            out.append((gu.read(f, "IRRADIANCE_HISTORY", P * 256, np.float32), gu.read(f, "DEPTH_HISTORY", P * 128, np.float32)))
        finally:
            f.dispose()
    for a, b in zip(*out):
        assert gu.texel_rel_err(a, b).max() <= gu.TEXEL_REL
