"""A solve captured into a caller's CUDA graph (the stages' dependent launches, the
cursors that each solve leaves clear): replays among ordinary solves give bit for bit
what ordinary solves alone give."""
import ctypes as C

import numpy as np
import pytest

from speedball_b200 import _abi, synth

import gpu_util as gu

pytestmark = pytest.mark.gpu


def _state(f):
    P = f._probeTotal
    return np.concatenate([gu.read(f, "IRRADIANCE_HISTORY", P * 256, np.float32),
                           gu.read(f, "DEPTH_HISTORY", P * 128, np.float32)])


@pytest.mark.parametrize("emitters", [False, True])
def test_captured_solves_among_ordinary_ones(emitters):
    torch = pytest.importorskip("torch")
    out = []
    for captured in (False, True):
        scene = synth.room_spheres(5)
        if emitters:
            scene = synth.add_emitters(scene)
        scene.meta["grid"] = dict(scene.meta["grid"], res=(5, 4, 3))
        f = gu.make_field(scene)
        try:
            f.tick()
            f.synchronize()
            P = f._probeTotal
            stream = torch.cuda.Stream()
            _abi.check(f._lib.sb_set_stream(f.ctx, C.c_void_p(stream.cuda_stream)), f.ctx)

            def solve():
                _abi.check(f._lib.sb_solve(f.ctx, 0, 0, P), f.ctx)
            solve()
            f.synchronize()
            if captured:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=stream):
                    solve()
            with torch.cuda.stream(stream):
                for k in range(4):
                    if captured and k != 2:
                        graph.replay()
                    else:
                        solve()
            f.synchronize()
            out.append(_state(f))
        finally:
            f.dispose()
    assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))
