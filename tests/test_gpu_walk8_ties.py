"""Equal hits in the warp walks. The lanes of a warp share their last rays, so the items
of one ray are met in no fixed order; the hit is still that of a walk by itself. Every
sphere of the room stands twice at the same place, so each hit on one is a tie of two
instances with equal bits of t: a ray names the same triangle and instance alone, in
company and in another order, and the t of the two-level walk."""
import ctypes as C

import numpy as np
import pytest

from speedball_b200 import _abi, synth
from speedball_b200.scene import Instance

import gpu_util as gu

pytestmark = pytest.mark.gpu


def _cast(f, ro, rd):
    n = len(ro)
    ro, rd = np.ascontiguousarray(ro), np.ascontiguousarray(rd)
    t, tri, inst = np.zeros(n, np.float32), np.zeros(n, np.int32), np.zeros(n, np.int32)
    _abi.check(f._lib.sb_raycast(f.ctx, _abi.ptr(ro), _abi.ptr(rd), n, _abi.ptr(t), _abi.ptr(tri), _abi.ptr(inst)), f.ctx)
    return t, tri, inst


def _kind(f, kind):
    t = _abi.sb_tuning()
    _abi.check(f._lib.sb_get_tuning(f.ctx, C.byref(t)), f.ctx)
    t.bvhKind = kind
    _abi.check(f._lib.sb_set_tuning(f.ctx, C.byref(t)), f.ctx)


@pytest.mark.parametrize("moved", [False, True])
def test_ties_do_not_depend_on_the_company(moved):
    s = synth.room_spheres(6)
    s.instances += [Instance(i.mesh, i.world.copy()) for i in s.instances[1:]]
    f = gu.make_field(s, record=False)
    try:
        f.tick()
        if moved:  # one of a pair leaves the tree without leaving its place, another pair moves
            for i in (3, 10, 74):
                s.instances[i].world = s.instances[i].world @ synth.trs((0.0 if i == 3 else 0.25, 0.0, 0.0))
            f.markTransformsDirty([3, 10, 74])
            f.tick()
        f.synchronize()
        rng = np.random.default_rng(8)
        n = 3000
        ro = rng.uniform(0.2, 9.8, (n, 3)).astype(np.float32)
        rd = rng.normal(size=(n, 3)).astype(np.float32)
        rd /= np.linalg.norm(rd, axis=1, keepdims=True)
        all_ = _cast(f, ro, rd)
        for size in (1, 5, 40):
            for a in range(0, 200, size):
                got = _cast(f, ro[a:a + size], rd[a:a + size])
                for x, y in zip(got, all_):
                    assert np.array_equal(x, y[a:a + size])
        order = rng.permutation(n)
        for x, y in zip(_cast(f, ro[order], rd[order]), all_):
            assert np.array_equal(x, y[order])
        _kind(f, 0)
        t, tri, inst = _cast(f, ro, rd)
        same = (tri == all_[1]) & (inst == all_[2])
        assert np.array_equal(t[same], all_[0][same])
        assert np.all(np.abs(t - all_[0])[~same] <= gu.TIE_REL * np.abs(t)[~same])
        assert 0.5 < (tri >= 0).mean()
    finally:
        f.dispose()
