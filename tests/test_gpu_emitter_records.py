"""Emitter visibility beside next-event estimation. A record of the emitter range that a
later sb_upload_range makes a point light is both: its visibility history is the one of the
emitter, and every ray's tested and unblocked lights are those of the point light, as if
each stood alone (bit for bit: the walks decide the same rays)."""
import ctypes as C

import numpy as np
import pytest

from speedball_b200 import _abi, synth

import gpu_util as gu

pytestmark = pytest.mark.gpu


def _field():
    s = synth.add_emitters(synth.room_spheres(0))
    s.meta["grid"] = dict(s.meta["grid"], res=(6, 5, 4))
    f = gu.make_field(s)
    f.tick()
    f.synchronize()
    return f


def _solved(f):
    P, n = f._probeTotal, f._probeTotal * f.getRays()
    for offset, count in ((0, P), (P - 7, 20)):
        _abi.check(f._lib.sb_solve(f.ctx, 0, offset, count), f.ctx)
        f.synchronize()
    vis = gu.read(f, "VISIBILITY", n * 4, np.uint32).reshape(-1, 4)
    return vis, gu.read(f, "EMITTER_VIS", P * 16, np.float32).reshape(P, 16)


def test_a_light_in_the_emitter_range():
    fields = [_field() for _ in range(3)]
    try:
        emitters, both, light = fields
        n, base = both._lightCount, both._lightCount - 3
        at = (base + 1) * 17
        one = np.ones(1, np.float32)
        _abi.check(both._lib.sb_upload_range(both.ctx, _abi.BUF["LIGHTS"], at, 1, _abi.ptr(one)), both.ctx)
        recs = gu.read(light, "LIGHTS", n * 17, np.float32)
        recs[at] = 1.0
        _abi.check(light._lib.sb_upload_lights(light.ctx, _abi.ptr(recs), n, 0, 0, 0), light.ctx)
        _, evis = _solved(emitters)
        got_vis, got_evis = _solved(both)
        vis, _ = _solved(light)
        bit = np.uint32(1 << (base + 1))
        assert 0.1 < ((vis[:, 0] & bit) != 0).mean() and 0.0 < evis[:, 1].mean() < 1.0
        assert np.array_equal(got_vis, vis)
        assert np.array_equal(got_evis, evis)
    finally:
        for f in fields:
            f.dispose()
