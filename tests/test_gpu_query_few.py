"""Queries of few rays: one launch on every layout of the scene (a second one, for the hits'
parameters, for the moved slots or to clear a cursor, doubled the time of a handful of rays);
and the same hits, bit for bit, whichever way a query of its size goes."""
import ctypes as C

import numpy as np
import pytest

from speedball_b200 import _abi, synth

import gpu_util as gu

pytestmark = pytest.mark.gpu

FEW = 1 << 18  # from here on the warps share the rays by a cursor


@pytest.mark.parametrize("kind", [1, 2, 0])
@pytest.mark.parametrize("moved", [0, 3])
def test_few_rays(kind, moved):
    torch = pytest.importorskip("torch")
    f = gu.make_field(synth.room_spheres(2), record=False)
    try:
        t = _abi.sb_tuning()
        _abi.check(f._lib.sb_get_tuning(f.ctx, C.byref(t)), f.ctx)
        t.bvhKind = kind
        _abi.check(f._lib.sb_set_tuning(f.ctx, C.byref(t)), f.ctx)
        f.tick()
        if moved:
            f.markTransformsDirty(list(range(1, 1 + moved)))
            f.tick()
        f.synchronize()
        n = FEW + 1
        rng = np.random.default_rng(kind)
        rd = rng.normal(size=(n, 3))
        rays = (rng.uniform(0.2, 9.8, (n, 3)), rd / np.linalg.norm(rd, axis=1, keepdims=True), rng.uniform(0, 8, n))
        ro, rd, dist = (torch.from_numpy(x.astype(np.float32)).cuda() for x in rays)
        out = [torch.empty(n, dtype=d, device="cuda") for d in (torch.int32, torch.int32, torch.int32, torch.uint8)]
        p = lambda x: C.c_void_p(x.data_ptr())  # noqa: E731
        torch.cuda.synchronize()

        def launched():
            st = _abi.sb_stats()
            _abi.check(f._lib.sb_get_stats(f.ctx, C.byref(st)), f.ctx)
            return st.kernelLaunches

        def cast(a, b):
            """Rays [a, b): the outputs and each query's launches."""
            for o in out:
                o.fill_(77)
            torch.cuda.synchronize()
            l0 = launched()
            _abi.check(f._lib.sb_raycast_device(f.ctx, p(ro[a:b]), p(rd[a:b]), b - a, *(p(o) for o in out[:3])), f.ctx)
            l1 = launched()
            _abi.check(f._lib.sb_occluded_device(f.ctx, p(ro[a:b]), p(rd[a:b]), p(dist[a:b]), b - a, p(out[3])), f.ctx)
            l2 = launched()
            f.synchronize()
            assert all((o[b - a:] == 77).all() for o in out)
            return [o[:b - a].cpu().numpy() for o in out], (l1 - l0, l2 - l1)
        want, _ = cast(0, n)
        assert (want[1] >= 0).mean() > 0.9 and 0.1 < want[3].mean() < 0.9
        for a, b in ((0, 1), (5, 36), (40, 73), (100, 10_100), (1, FEW), (0, FEW)):
            got, launches = cast(a, b)
            for g, w in zip(got, want):
                assert np.array_equal(g, w[a:b]), (a, b)
            if b - a < FEW:
                assert launches == (1, 1), (a, b, launches)
    finally:
        f.dispose()
