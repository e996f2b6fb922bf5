"""Queries share nothing but the scene: closest hits and occlusion enqueued on two streams
without an order between them, and captured queries replayed side by side, write every ray
of each, bit for bit what they write one after the other."""
import ctypes as C

import numpy as np
import pytest

from speedball_b200 import _abi, synth

import gpu_util as gu

pytestmark = pytest.mark.gpu

RAYS = 600_011


@pytest.mark.parametrize("captured,moved", [(False, False), (True, False), (False, True), (True, True)])
def test_queries_on_two_streams(captured, moved):
    torch = pytest.importorskip("torch")
    f = gu.make_field(synth.room_spheres(4))
    try:
        f.tick()
        if moved:
            f.markTransformsDirty([3, 17, 40])
            f.tick()
        f.synchronize()
        n = 100_003 if moved else RAYS  # with moved slots: by walk2 too
        rng = np.random.default_rng(1)
        streams = [torch.cuda.Stream() for _ in range(2)]
        jobs = []
        for k in range(2):
            ro = rng.uniform(0.2, 9.8, (n, 3)).astype(np.float32)
            rd = rng.normal(size=(n, 3)).astype(np.float32)
            rd /= np.linalg.norm(rd, axis=1, keepdims=True)
            ins = [torch.from_numpy(x).cuda() for x in (ro, rd, rng.uniform(0, 8, n).astype(np.float32))]
            outs = [torch.empty(n, dtype=d, device="cuda") for d in (torch.float32, torch.int32, torch.int32, torch.uint8)]
            jobs.append((ins, outs))
        p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731

        def enqueue(k):
            (ro, rd, dist), (t, tri, inst, occ) = jobs[k]
            _abi.check(f._lib.sb_set_stream(f.ctx, C.c_void_p(streams[k].cuda_stream)), f.ctx)
            _abi.check(f._lib.sb_raycast_device(f.ctx, p(ro), p(rd), n, p(t), p(tri), p(inst)), f.ctx)
            _abi.check(f._lib.sb_occluded_device(f.ctx, p(ro), p(rd), p(dist), n, p(occ)), f.ctx)

        def results():
            torch.cuda.synchronize()
            out = [[o.cpu().numpy().copy() for o in outs] for _, outs in jobs]
            for _, outs in jobs:
                for o in outs:
                    o.fill_(77)
            torch.cuda.synchronize()
            return out
        results()
        for k in range(2):
            enqueue(k)
            torch.cuda.synchronize()
        want = results()
        assert all((w[1] >= 0).mean() > 0.9 for w in want)
        graphs = []
        if captured:
            for k in range(2):
                graphs.append(torch.cuda.CUDAGraph())
                with torch.cuda.graph(graphs[k], stream=streams[k]):
                    enqueue(k)
        for _ in range(5):
            for k in range(2):
                if captured:
                    with torch.cuda.stream(streams[k]):
                        graphs[k].replay()
                else:
                    enqueue(k)
            for got, exp in zip(results(), want):
                for a, b in zip(got, exp):
                    assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    finally:
        f.dispose()
