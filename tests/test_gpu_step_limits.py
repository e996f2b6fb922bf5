"""Step limits with moved slots: sb_set_walk_step_limit holds for a ray's walk of the tree and
of each moved slot's BLAS by itself, so a limit of a mesh's whole node count cannot run
out in its slots, however many of them a ray meets."""
import numpy as np
import pytest

from speedball_b200 import _abi, synth
from speedball_b200.scene import Instance

import gpu_util as gu

pytestmark = pytest.mark.gpu


def test_a_limit_holds_for_each_moved_slot():
    s = synth.room_spheres(0)
    s.instances = s.instances[:1] + [Instance(1, synth.trs((5.0 + 0.001 * k, 5.0, 5.0), s=4.0)) for k in range(40)]
    s.meta["grid"] = dict(s.meta["grid"], gridMin=(0.5, 0.5, 0.5), gridSize=(9.0, 9.0, 9.0), res=(3, 3, 3))
    f = gu.make_field(s)
    try:
        f.tick()
        f.markTransformsDirty(list(range(1, 41)))
        f.tick()
        f.synchronize()
        P = f._probeTotal
        n = P * f.getRays()

        def hits():
            _abi.check(f._lib.sb_solve(f.ctx, 0, 0, P), f.ctx)
            f.synchronize()
            return gu.read(f, "HIT_RECORDS", n * 4, np.uint32)
        want = hits()
        pool = f.pool
        _abi.check(f._lib.sb_set_walk_step_limit(f.ctx, int(pool.blas_end[1] - pool.blas_root[1])), f.ctx)
        assert np.array_equal(hits(), want)
        _abi.check(f._lib.sb_set_walk_step_limit(f.ctx, 8), f.ctx)
        with pytest.raises(_abi.SbError):  # a limit that does run out is reported
            hits()
    finally:
        f.dispose()
