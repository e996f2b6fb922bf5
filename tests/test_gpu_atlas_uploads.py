"""Ranged uploads into the atlases: the receivers' layout follows each range, whatever its
ends, and no more of it than the rows of probes the range touches. Parts of every kind in any
order give the receivers what one upload of the whole gives (bit for bit), and an upload
of one texel's word costs a field of 32^3 probes no more than one of 4^3 (within 2)."""
import ctypes as C

import numpy as np
import pytest

from speedball_b200 import _abi, synth

import gpu_util as gu

pytestmark = pytest.mark.gpu


def _field(res):
    s = synth.room_spheres(1)
    s.meta["grid"] = dict(s.meta["grid"], res=res)
    return gu.make_field(s)


def _upload(f, which, flat, a, b):
    part = np.ascontiguousarray(flat[a:b])
    _abi.check(f._lib.sb_upload_range(f.ctx, _abi.BUF[which], a, b - a, _abi.ptr(part)), f.ctx)


def _gathered(f, torch):
    rng = np.random.default_rng(1)
    g = f.grid
    n = 4000
    p4, n4 = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    p4[:, :3] = np.array(g.gridMin) + np.array(g.gridSize) * rng.random((n, 3))
    n4[:, :3] = rng.normal(size=(n, 3))
    prm = _abi.sb_gather_params()
    f._lib.sb_gather_params_defaults(C.byref(prm))
    prm.chebyStrength = 0.75
    dev = [torch.from_numpy(a).cuda() for a in (p4, n4)] + [torch.zeros(n, 4, device="cuda")]
    torch.cuda.synchronize()
    p = [C.c_void_p(t.data_ptr()) for t in dev]
    _abi.check(f._lib.sb_gather_irradiance(f.ctx, C.byref(prm), p[0], p[1], p[1], n, p[2]), f.ctx)
    f.synchronize()
    return dev[2].cpu().numpy()


@pytest.mark.parametrize("res", [(2, 2, 2), (5, 3, 4)])
def test_parts_give_what_the_whole_gives(res):
    torch = pytest.importorskip("torch")
    whole, parts = _field(res), _field(res)
    try:
        rng = np.random.default_rng(sum(res))
        size = res[0] * 8 * res[1] * res[2] * 8 * 4
        data = dict(IRRADIANCE_ATLAS=rng.uniform(0.1, 4.0, size).astype(np.float16),
                    DEPTH_ATLAS=rng.uniform(0.5, 3.0, size).astype(np.float16))
        for which, flat in data.items():
            _upload(whole, which, flat, 0, size)
            row = res[0] * 8 * 4 * 8  # a row of tiles
            ends = {0, 1, row - 1, row, row + 5, size - row, size - 1, size}
            ends = sorted(ends | set(int(x) for x in rng.integers(0, size, 12)))
            for k in rng.permutation(len(ends) - 1):
                _upload(parts, which, flat, ends[k], ends[k + 1])
        a, b = _gathered(whole, torch), _gathered(parts, torch)
        assert np.abs(a[:, :3]).max() > 0.1
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    finally:
        whole.dispose()
        parts.dispose()


def test_a_small_part_of_a_large_field():
    torch = pytest.importorskip("torch")
    times = []
    for res in ((4, 4, 4), (32, 32, 32)):
        f = _field(res)
        try:
            stream = torch.cuda.Stream()
            _abi.check(f._lib.sb_set_stream(f.ctx, C.c_void_p(stream.cuda_stream)), f.ctx)
            one = torch.ones(1, dtype=torch.float16).pin_memory()

            def uploads(n):
                for k in range(n):
                    which = _abi.BUF["IRRADIANCE_ATLAS" if k % 2 else "DEPTH_ATLAS"]
                    _abi.check(f._lib.sb_upload_range(f.ctx, which, 0, 1, C.c_void_p(one.data_ptr())), f.ctx)
            uploads(20)
            best = float("inf")
            for _ in range(5):
                a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                with torch.cuda.stream(stream):
                    torch.cuda._sleep(5_000_000)  # all are enqueued before the first runs
                a.record(stream)
                uploads(100)
                b.record(stream)
                b.synchronize()
                best = min(best, a.elapsed_time(b))
            times.append(best)
        finally:
            f.dispose()
    print(times)
    assert times[1] <= 2.0 * times[0], times
