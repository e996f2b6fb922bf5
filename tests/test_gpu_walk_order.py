"""Which of two hits of one t a warp walk names. The lanes of a warp share their last rays
and test the items in rounds, so two items of equal t from different leaves meet in
different rounds and in any order; the hit is still the first in the order of a walk by
itself. Planes of small triangles, each with one of two large triangles in the same
place: a vertical ray meets a small and a large one at the same exact t, in distant leaves.
It names the same triangle and instance alone, among 5, among 40, in one large launch, and
in walks that share nothing (a step limit below the default). Slots that have moved,
walked through their own BLAS ahead of the tree, the same for the rays of one probe, of
all, and of walks that share nothing. Every launch does the same arithmetic on a ray: no
tolerance."""
import ctypes as C

import numpy as np
import pytest

from speedball_b200 import _abi, synth
from speedball_b200.scene import Instance, Mesh, SceneDesc

import gpu_util as gu

pytestmark = pytest.mark.gpu

NO_SHARING = (1 << 26) - 1  # a step limit below the walks' default: each lane walks its rays by itself


def _plane(n):
    """n x n squares over [-2, 2]^2 in y = 0."""
    P, F = synth.grid_mesh(n, n, lambda u, v: (4 * u - 2, 0 * u, 4 * v - 2))
    return P, F


def _merged(parts, seed):
    Ps, Fs, n = [], [], 0
    for P, F in parts:
        Ps.append(P)
        Fs.append(F + n)
        n += len(P)
    F = np.random.default_rng(seed).permutation(np.concatenate(Fs)).astype(np.uint32)
    return Mesh(np.concatenate(Ps), F, np.zeros(len(F), np.uint32))


def _scene(seed):
    """A room with six planes, each once small and once large: two meshes of one place, or one of both."""
    s = synth.room_spheres(seed)
    rng = np.random.default_rng(seed)
    s.instances = s.instances[:1 + 8 * (seed % 3)]
    first = len(s.instances)
    s.meshes = list(s.meshes)
    for k in range(6):
        n, at = (8, 16, 32, 64)[rng.integers(4)], synth.trs((4.0 + k % 3, 1.0 + 1.25 * k, 4.0 + k % 2))
        parts = [_plane(n), _plane(1)]
        if k % 2:
            s.meshes.append(_merged(parts, seed))
            s.instances.append(Instance(len(s.meshes) - 1, at))
        else:
            for i in rng.permutation(2):
                s.meshes.append(_merged([parts[i]], seed))
                s.instances.append(Instance(len(s.meshes) - 1, at))
    return s, first


def _cast(f, ro, rd):
    n = len(ro)
    ro, rd = np.ascontiguousarray(ro), np.ascontiguousarray(rd)
    t, tri, inst = np.zeros(n, np.float32), np.zeros(n, np.int32), np.zeros(n, np.int32)
    _abi.check(f._lib.sb_raycast(f.ctx, _abi.ptr(ro), _abi.ptr(rd), n, _abi.ptr(t), _abi.ptr(tri), _abi.ptr(inst)), f.ctx)
    return np.stack([t.view(np.int32), tri, inst], 1)


def _rays(n, seed):
    """Vertical rays inside the planes' smallest triangles, up and down, at multiples of 1/32."""
    rng = np.random.default_rng(seed)
    ro = np.empty((n, 3), np.float32)
    cell = rng.integers(0, 48, (2, n))
    ro[:, 0] = 2.0 + cell[0] / 8.0 + 1 / 16
    ro[:, 2] = 2.0 + cell[1] / 8.0 + 1 / 32
    ro[:, 1] = rng.integers(1, 38, n) / 4.0 + 1 / 8
    rd = np.zeros((n, 3), np.float32)
    rd[:, 1] = np.where(rng.random(n) < 0.5, 1.0, -1.0)
    return ro, rd


@pytest.mark.parametrize("seed,moved", [(1, False), (2, False), (3, True), (7, False)])
def test_hits_of_equal_t_do_not_depend_on_the_company(seed, moved):
    s, first = _scene(seed)
    f = gu.make_field(s, record=False)
    try:
        f.tick()
        if moved:  # some leave the tree without leaving their place
            f.markTransformsDirty([first, first + 2, first + 5])
            f.tick()
        f.synchronize()
        n = 3_000
        ro, rd = _rays(n, seed)
        rng = np.random.default_rng(9)
        fro = rng.uniform(0.2, 9.8, (270_000, 3)).astype(np.float32)
        frd = rng.normal(size=(270_000, 3)).astype(np.float32)
        frd /= np.linalg.norm(frd, axis=1, keepdims=True)
        _abi.check(f._lib.sb_set_walk_step_limit(f.ctx, NO_SHARING), f.ctx)
        want = _cast(f, ro, rd)
        assert len(np.unique(want[:, 2])) > 6
        _abi.check(f._lib.sb_set_walk_step_limit(f.ctx, 0), f.ctx)
        bad = {}  # rays whose hit is another, per launch
        got = _cast(f, np.concatenate([ro, fro]), np.concatenate([rd, frd]))[:n]
        bad["large"] = int((got != want).any(1).sum())
        for size in (1, 2, 12, 40, n):
            got = np.concatenate([_cast(f, ro[a:a + size], rd[a:a + size]) for a in range(0, n, size)])
            bad[size] = int((got != want).any(1).sum())
        for k in range(4):
            p = rng.permutation(n)
            bad["order", k] = int((_cast(f, ro[p], rd[p]) != want[p]).any(1).sum())
        assert not any(bad.values()), bad
    finally:
        f.dispose()


@pytest.mark.parametrize("seed,moved", [(0, False), (1, True), (4, True)])
def test_probe_rays_of_equal_t_do_not_depend_on_the_company(seed, moved):
    s, first = _scene(seed)
    s.meta["grid"] = dict(s.meta["grid"], res=(4, 6, 4), rays=128)
    f = gu.make_field(s)
    try:
        f.tick()
        if moved:
            f.markTransformsDirty(list(range(first, len(s.instances))))
            f.tick()
        f.synchronize()
        P, R = f._probeTotal, f.getRays()

        def hits(offset, count):
            _abi.check(f._lib.sb_solve(f.ctx, 0, offset, count), f.ctx)
            f.synchronize()
            return gu.read(f, "HIT_RECORDS", count * R * 4, np.uint32).reshape(-1, 4)
        _abi.check(f._lib.sb_set_walk_step_limit(f.ctx, NO_SHARING), f.ctx)
        want = hits(0, P)
        assert (want[:, 0] != 0xFFFFFFFF).mean() > 0.9
        alone = np.concatenate([hits(p, 1) for p in range(P)])
        bad = {"alone, nothing shared": int((alone != want).any(1).sum())}
        _abi.check(f._lib.sb_set_walk_step_limit(f.ctx, 0), f.ctx)
        for k in range(4):
            bad[k] = int((hits(0, P) != want).any(1).sum())
        bad["probes"] = int((np.concatenate([hits(p, 1) for p in range(P)]) != want).any(1).sum())
        assert not any(bad.values()), bad
    finally:
        f.dispose()


def test_moved_ties_name_the_first_slot_and_lowest_triangle():
    """A ball whose triangles stand three times over, twice in one place, moved: of the six
    equal hits a ray names the first listed slot's lowest triangle (the reference's order)."""
    s, _ = _scene(0)
    P, F, _ = synth.icosphere(2, 1.5)
    F = np.random.default_rng(1).permutation(np.repeat(F, 3, 0)).astype(np.uint32)
    s.meshes.append(Mesh(P, F, np.zeros(len(F), np.uint32)))
    first = len(s.instances)
    s.instances += [Instance(len(s.meshes) - 1, synth.trs((2.5, 7.5, 7.5))) for _ in range(2)]
    s.meta["grid"] = dict(s.meta["grid"], res=(4, 6, 4), rays=128)
    f = gu.make_field(s)
    try:
        f.tick()
        f.markTransformsDirty([first, first + 1])
        f.tick()
        f.synchronize()
        P, R = f._probeTotal, f.getRays()
        _abi.check(f._lib.sb_solve(f.ctx, 0, 0, P), f.ctx)
        f.synchronize()
        hits = gu.read(f, "HIT_RECORDS", P * R * 4, np.uint32).reshape(-1, 4)
        order = gu.read(f, "TLAS_ORDER", len(s.instances), np.uint32)
        slots = [int(np.flatnonzero(order == first + k)[0]) for k in range(2)]
        tri, slot = hits[:, 0], hits[:, 1] & 0x7FFFFFFF
        on = np.isin(slot, slots) & (tri != 0xFFFFFFFF)
        assert on.sum() > 100 and np.array_equal(np.unique(slot[on]), slots[:1])
        corners = np.sort(f.pool.triIndex.reshape(-1, 3), 1)
        _, group = np.unique(corners, axis=0, return_inverse=True)
        lowest = np.full(group.max() + 1, len(group))
        np.minimum.at(lowest, group, np.arange(len(group)))
        assert np.array_equal(lowest[group[tri[on]]], tri[on])
    finally:
        f.dispose()


def _kind(f, kind):
    t = _abi.sb_tuning()
    _abi.check(f._lib.sb_get_tuning(f.ctx, C.byref(t)), f.ctx)
    t.bvhKind = kind
    _abi.check(f._lib.sb_set_tuning(f.ctx, C.byref(t)), f.ctx)


@pytest.mark.parametrize("seed", [1, 2])
def test_moved_queries_name_the_hits_of_one_thread_a_ray(seed):
    """Every plane moved. By the warps' walk (few rays), one thread per ray (from 2^18) and
    beside the binary tree, whose rays each walk the moved slots in the reference's order: the
    same triangle, instance and t of two that are as near, and the same rays blocked."""
    s, first = _scene(seed)
    f = gu.make_field(s, record=False)
    try:
        f.tick()
        f.markTransformsDirty(list(range(first, len(s.instances))))
        f.tick()
        f.synchronize()
        n, large = 3_000, (1 << 18) + 5
        ro, rd = _rays(n, seed)
        at = np.arange(large) % n

        def occluded(ro, rd):
            out = np.zeros(len(ro), np.uint8)
            dist = np.full(len(ro), 2.0, np.float32)
            _abi.check(f._lib.sb_occluded(f.ctx, _abi.ptr(ro), _abi.ptr(rd), _abi.ptr(dist), len(ro), _abi.ptr(out)), f.ctx)
            return out
        got, occ = _cast(f, ro, rd), occluded(ro, rd)
        assert np.array_equal(_cast(f, ro[at], rd[at]), got[at])
        assert np.array_equal(occluded(ro[at], rd[at]), occ[at])
        _kind(f, 2)
        _abi.check(f._lib.sb_rebuild_scene_bvh(f.ctx), f.ctx)
        f.tick()
        f.markTransformsDirty(list(range(first, len(s.instances))))
        f.tick()
        f.synchronize()
        assert np.array_equal(_cast(f, ro, rd), got) and np.array_equal(occluded(ro, rd), occ)
        assert 0.1 < occ.mean() < 0.9
    finally:
        f.dispose()
