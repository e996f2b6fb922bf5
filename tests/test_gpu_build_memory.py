"""The BLAS builder's scratch follows the mesh: sixteen contexts that each build a mesh of
700 triangles take 64 KB each, so no more than two of the driver's 2 MB blocks together
(one that has to be mapped makes a context's first build wait for some 350 us); a mesh of
rising size after it builds the same tree as in a context of its own."""
import ctypes as C

import numpy as np
import pytest

from speedball_b200 import _abi, synth

pytestmark = pytest.mark.gpu


def _context():
    lib, ctx = _abi.load(), C.c_void_p()
    _abi.check(lib.sb_create(C.byref(_abi.sb_device_opts(0, 0)), C.byref(ctx)))
    return lib, ctx


def _build(lib, ctx, tris, torch):
    P, F = synth.column_prism(tris, np.random.default_rng(tris))
    pos = torch.from_numpy(np.ascontiguousarray(P, np.float32)).cuda()
    idx = torch.from_numpy(np.ascontiguousarray(F).astype(np.int32)).cuda()
    T = len(F)
    out = [torch.zeros(n, dtype=torch.int32, device="cuda") for n in (16 * T, T, 1)]
    torch.cuda.synchronize()

    def run():
        p = [C.c_void_p(t.data_ptr()) for t in (pos, idx, *out)]
        _abi.check(lib.sb_build_blas_device(ctx, p[0], len(P), p[1], T, 8, p[2], p[3], p[4]), ctx)
        _abi.check(lib.sb_synchronize(ctx), ctx)
        return [t.cpu().numpy() for t in out]
    return run


def test_scratch_of_small_builds():
    torch = pytest.importorskip("torch")
    contexts = [_context() for _ in range(16)]
    try:
        runs = [_build(lib, ctx, 700, torch) for lib, ctx in contexts]
        free = torch.cuda.mem_get_info()[0]
        trees = [run() for run in runs]
        assert free - torch.cuda.mem_get_info()[0] <= 4 << 20
        for t in trees[1:]:
            assert all(np.array_equal(a, b) for a, b in zip(t, trees[0]))
    finally:
        for lib, ctx in contexts:
            lib.sb_destroy(ctx)


def test_meshes_of_rising_and_falling_size():
    torch = pytest.importorskip("torch")
    lib, ctx = _context()
    try:
        for tris in (40, 700, 1_500, 9_000, 5_000, 60_000, 200_000, 700):
            got = _build(lib, ctx, tris, torch)()
            l1, c1 = _context()
            want = _build(l1, c1, tris, torch)()
            l1.sb_destroy(c1)
            assert all(np.array_equal(a, b) for a, b in zip(got, want)), tris
    finally:
        lib.sb_destroy(ctx)
