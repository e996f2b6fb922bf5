"""The parameter sums of the shading adjoint: a warp's rays put their material's terms into
the warp's table and the first ray of each material reads them back. From one material
in the whole scene, which all lanes share, to more than a warp's lanes, against the FP64
adjoint on the GPU's own records at the bar of the other gradient tests (1e-3 relative,
floor 1e-5 of the largest).

With more entries than the shared table holds, the sums are formed in FP64 throughout, so
a gradient does not depend on how its terms are grouped beyond its own rounding to FP32:
rays taken out of one material into another of the same record leave what the second one
gains, also where the terms of either sign all but cancel (tolerance: the three results'
roundings, and 1e-12 of the sum of the terms' sizes for the FP64 sums)."""
import numpy as np
import pytest

from speedball_b200 import synth
from speedball_b200.adjoint import GIAdjoint

from gpu_util import OracleMirror, gpu_records, make_field

pytestmark = pytest.mark.gpu


def _flat(g):
    return np.concatenate([g["albedo"].reshape(-1), g["emissive"].reshape(-1), g["lightScale"].reshape(-1)])


@pytest.mark.parametrize("materials,lights", [(1, 1), (2, 7), (40, 33)])
def test_sums_over_shared_materials(materials, lights, orc):
    s = synth.room_spheres(3, n_materials=materials, n_point=lights, n_dir=0)
    s.meta["grid"] = dict(s.meta["grid"], res=(5, 4, 3), rays=48)
    f = make_field(s)
    try:
        adj = GIAdjoint(f, solves=1)
        E = adj.forward()
        target = (E * np.random.default_rng(1).uniform(0.5, 1.5, E.shape)).astype(np.float32)
        adj.forward(target)
        got = _flat(adj.backward())
        mirror = OracleMirror(f)
        rec = gpu_records(f, adj.probes * f.getRays())
        base = adj.parameters()
        _, _, want = orc.adjoint(mirror.scene, mirror.arena, mirror.light_count, mirror.clustered, mirror.grid,
                                 mirror.params(), rec["tri"], rec["inst_word"], rec["blocked"], 1,
                                 base["albedo"].astype(np.float32).astype(np.float64).reshape(-1),
                                 base["emissive"].reshape(-1), np.ones(lights),
                                 target=target.astype(np.float64).reshape(-1), round_atlas=True)
        scale = np.abs(want).max()
        assert (np.abs(got - want) <= 1e-3 * np.abs(want) + 1e-5 * scale).all()
    finally:
        f.dispose()


def _one_or_two_materials(two):
    s = synth.room_spheres(3, n_materials=1400, n_point=3, n_dir=0)
    s.materials[:] = s.materials[0]
    for m in s.meshes:
        m.tri_material[:] = 0
    if two:
        s.meshes[9].tri_material[::16] = 1
    s.meta["grid"] = dict(s.meta["grid"], res=(6, 6, 6))
    return s


@pytest.mark.parametrize("seed", [0, 1, 3])
def test_sums_in_fp64_with_many_materials(seed):
    fields = [make_field(_one_or_two_materials(two), record=False) for two in (False, True)]
    try:
        one, two = (GIAdjoint(f, solves=1) for f in fields)
        assert 6 * one.materialCount + one.lightCount > 8192
        E = one.forward()
        assert np.array_equal(E, two.forward())
        rng = np.random.default_rng(seed)
        n1, n2 = (E * rng.choice([-1.0, 1.0], E.shape) for _ in range(2))

        def gradient(a, noise):
            a.forward((E - noise).astype(np.float32))
            return a.backward()["emissive"].astype(np.float64)
        a, b = gradient(one, n1)[0, 0], gradient(one, n2)[0, 0]
        size = np.abs(gradient(one, np.abs(n1)))[0, 0]  # terms of one sign: the sum of their sizes, about
        noise = n1 - a / b * n2
        whole, parts = gradient(one, noise), gradient(two, noise)
        g, g0, g1 = whole[0, 0], parts[0, 0], parts[1, 0]
        assert abs(g) < 1e-3 * size and g1 != 0.0
        assert abs(g - (g0 + g1)) <= 2.0 ** -24 * (abs(g) + abs(g0) + abs(g1)) + 1e-12 * size, (g, g0, g1, size)
    finally:
        for f in fields:
            f.dispose()
