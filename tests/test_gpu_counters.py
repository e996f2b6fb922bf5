"""The visit counters of the 8-wide walks. Each item test of the tree reads its instance's
rows, so without moved slots there are as many instance visits as triangle tests, in
solves and in batches of any length; a moved slot adds one visit per ray that enters it,
whatever its triangles' tests. Counts are whole numbers: no tolerance."""
import ctypes as C

import pytest

from speedball_b200 import _abi, synth

import gpu_util as gu

pytestmark = pytest.mark.gpu


def _counted(lead, run):
    lib = lead._lib
    _abi.check(lib.sb_enable_counters(lead.ctx, 1), lead.ctx)
    run()
    lead.synchronize()
    st = _abi.sb_stats()
    _abi.check(lib.sb_get_stats(lead.ctx, C.byref(st)), lead.ctx)
    _abi.check(lib.sb_enable_counters(lead.ctx, 0), lead.ctx)
    assert st.primaryRays and st.shadowRays and st.triangleTests
    return st


@pytest.mark.parametrize("count", [1, 2, 5])
def test_instance_visits_of_batches(count):
    fields = [gu.make_field(synth.room_spheres(k)) for k in range(count)]
    try:
        items = (_abi.sb_solve_item * count)()
        for f, i in zip(fields, items):
            f.tick()
            f.synchronize()
            i.ctx, i.cascade, i.probeOffset, i.updatedCount = f.ctx, 0, 0, f._probeTotal
        st = _counted(fields[0], lambda: _abi.check(fields[0]._lib.sb_solve_batch(items, count), fields[0].ctx))
        assert st.instanceVisits == st.triangleTests
        assert st.shadowInstanceVisits == st.shadowTriangleTests
    finally:
        for f in fields:
            f.dispose()


def test_instance_visits_of_moved_slots():
    s = synth.room_spheres(0)
    f = gu.make_field(s)
    try:
        f.tick()
        f.markTransformsDirty([5, 6])
        f.tick()
        f.synchronize()
        solve = lambda: _abi.check(f._lib.sb_solve(f.ctx, 0, 0, f._probeTotal), f.ctx)  # noqa: E731
        st = _counted(f, solve)
        # the two spheres' 1,280 triangles: more tests than rays that enter them
        assert st.triangleTests > st.instanceVisits
    finally:
        f.dispose()
