"""sb_get_stats waits for the context's own stream and no other, as a program that works on
the default stream beside it relies on; the stages' times add up to the solve's."""
import ctypes as C

import pytest

from speedball_b200 import _abi, synth

import gpu_util as gu

pytestmark = pytest.mark.gpu


def _stats(f):
    st = _abi.sb_stats()
    _abi.check(f._lib.sb_get_stats(f.ctx, C.byref(st)), f.ctx)
    return st


def test_stats_do_not_wait_for_other_streams():
    torch = pytest.importorskip("torch")
    f = gu.make_field(synth.room_spheres(0))
    try:
        f.tick()
        f.synchronize()
        torch.cuda.synchronize()
        st = _stats(f)
        stages = st.lastPrimaryMs + st.lastEmitMs + st.lastShadowMs + st.lastShadeMs
        assert 0.0 < st.lastTraceMs <= st.lastSolveMs
        assert min(st.lastPrimaryMs, st.lastEmitMs, st.lastShadowMs, st.lastShadeMs) > 0.0
        assert abs(stages - st.lastTraceMs) <= 1e-5  # sums of the same stamps, in FP32 milliseconds
        done = torch.cuda.Event()
        torch.cuda._sleep(1_000_000_000)  # half a second on the default stream
        done.record()
        again = _stats(f)
        assert not done.query()
        assert again.lastSolveMs == st.lastSolveMs and again.lastPrimaryMs == st.lastPrimaryMs
        torch.cuda.synchronize()
    finally:
        f.dispose()
