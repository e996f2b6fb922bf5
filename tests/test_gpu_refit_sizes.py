"""The refit lanes at the sizes where their paths change, bit for bit against the
oracle: meshes of one triangle, of one CTA's subtree, of a planned top and of more
subtrees than a plan holds; instance counts and updates on either side of a warp and
of a thread per instance and of the TLAS that fits shared memory."""
import numpy as np
import pytest

from speedball_b200 import synth
from speedball_b200.scene import Instance, Mesh

import gpu_util as gu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tris", [1, 2, 90, 350, 3_000, 30_000, 160_000])
def test_blas_refit(tris):
    rng = np.random.default_rng(tris)
    s = synth.room_spheres(0)
    n = max(2, int(np.ceil(np.sqrt(tris / 2))))
    P, F = synth.grid_mesh(n, n, lambda u, v: (2 + 6 * u, 5 + np.sin(9 * u) * np.cos(7 * v), 2 + 6 * v))
    F = F[:tris]
    s.meshes[7] = Mesh(P, F, np.zeros(len(F), np.uint32))
    f = gu.make_field(s, record=False)
    try:
        tail = gu.SceneTail(gu.OracleMirror(f))
        for _ in range(2):
            pos = (P + rng.normal(0, 0.05, P.shape)).astype(np.float32)
            s.meshes[7].positions = pos
            f.refreshDeforms([7])
            f.synchronize()
            tail.apply({7: pos}, {})
            tail.check_gpu()
    finally:
        f.dispose()


@pytest.mark.parametrize("count", [1, 2, 9, 48, 49, 300, 600])
def test_transform_lane(count):
    rng = np.random.default_rng(count)
    s = synth.room_spheres(0)
    s.instances = [Instance(1 + i % 64, synth.trs(rng.uniform(0, 10, 3))) for i in range(count)]
    f = gu.make_field(s, record=False)
    try:
        tail = gu.SceneTail(gu.OracleMirror(f))
        for k in sorted({1, min(8, count), min(48, count), count}):
            moved = {}
            for i in rng.choice(count, k, replace=False):
                m = synth.trs(rng.uniform(0, 10, 3), s=rng.uniform(0.2, 2.0))
                m[0, 1] = rng.normal()
                if i % 5 == 0:
                    m[2, :3] = 0.0  # no inverse
                s.instances[int(i)].world = m
                moved[int(i)] = m
            f.markTransformsDirty(list(moved))
            f._refresh_lanes()
            f.synchronize()
            tail.apply({}, moved)
            tail.check_gpu()
    finally:
        f.dispose()
