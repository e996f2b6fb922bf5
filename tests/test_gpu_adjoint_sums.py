"""The parameter sums of the shading adjoint: a warp's rays put their material's terms into
the warp's table and the first ray of each material reads them back. From one material
in the whole scene, which all lanes share, to more than a warp's lanes, against the FP64
adjoint on the GPU's own records at the bar of the other gradient tests (1e-3 relative,
floor 1e-5 of the largest)."""
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
