"""The emission stage's light gates (decided by squares from a table, with the exact
form for what lies near an edge) against the oracle's, on lights at the edges of the
gates: ranges of none, negative, tiny, huge and infinite, peaks of zero, negative and
subnormal, each type, a type past the last, the near-infrared class off and on. The
oracle shades the GPU's own hits in 64 bits. A gate may turn where FP32 rounding
reaches it: hit positions and normals carry 1e-5 of the room's size at most, so about
2e-5 of (ray, light) pairs lie that near to a range or a horizon; 1e-4 are allowed."""
import numpy as np
import pytest

from speedball_b200 import _abi, synth

import gpu_util as gu
import orc

pytestmark = pytest.mark.gpu


def _records():
    rng = np.random.default_rng(11)
    edge = [dict(), dict(range=-1.0), dict(range=4.0), dict(range=1e-6), dict(range=1e19), dict(range=np.inf),
            dict(col=(0, 0, 0)), dict(col=(-1, -2, -0.5)), dict(col=(0, 1e-40, 0)), dict(col=(1e-21, 0, 0)),
            dict(type=2, range=6.0), dict(type=0), dict(type=0, col=(0, 0, 0)), dict(type=3), dict(cls=4.0),
            dict(cls=4.0, type=0), dict(range=3.0), dict(type=2)]
    recs = np.zeros((len(edge), 17), np.float32)
    for r, e in zip(recs, edge):
        d = rng.normal(size=3)
        r[0] = e.get("type", 1)
        r[1:4] = rng.uniform(1.5, 8.5, 3)
        r[4:7] = d / np.linalg.norm(d)
        r[7:10] = e.get("col", (1.0, 0.5, 0.25))
        r[10], r[11], r[12], r[13], r[16] = e.get("range", 0.0), 2.0, 0.5, 0.9, e.get("cls", 0.0)
    return recs


@pytest.mark.parametrize("clustered,nir", [(False, 0.0), (False, 1.0), (True, 0.0)])
def test_gates_of_edge_lights(clustered, nir):
    scene = synth.room_spheres(3)
    scene.meta["grid"] = dict(scene.meta["grid"], res=(5, 4, 3))
    scene.meta["clustered"] = clustered
    f = gu.make_field(scene)
    try:
        f._params.nirGate = nir
        f.tick()
        f.synchronize()
        mirror = gu.OracleMirror(f)
        recs = _records()
        _abi.check(f._lib.sb_upload_lights(f.ctx, _abi.ptr(recs), len(recs), 0, 0, int(clustered)), f.ctx)
        mirror.arena = orc.light_arena(recs, clustered, mirror.g0dict)
        mirror.light_count = len(recs)
        P = f._probeTotal
        n = P * f.getRays()
        _abi.check(f._lib.sb_solve(f.ctx, 0, 0, P), f.ctx)
        f.synchronize()
        rec = gu.gpu_records(f, n)
        vis = gu.read(f, "VISIBILITY", n * 4, np.uint32).reshape(n, 4)
        tested = vis[:, 0].astype(np.uint64) | vis[:, 1].astype(np.uint64) << np.uint64(32)
        want = mirror.solve(0, P, replay=rec)["tested"]
        bits = np.arange(len(recs), dtype=np.uint64)
        got, want = ((x[:, None] >> bits & np.uint64(1)).astype(bool) for x in (tested, want))
        hits = int((rec["tri"] >= 0).sum())
        assert hits > n // 2 and 0.02 < want.mean() < 0.9
        differ = got != want
        assert differ.sum() <= 1e-4 * hits * len(recs), (int(differ.sum()), differ.sum(0))
    finally:
        f.dispose()
