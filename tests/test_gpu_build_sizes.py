"""The GPU BLAS build at the sizes where its paths change: a warp's and a tile's
edges (32, 1024 positions), clusters of 1, 2, 4 and 8 CTAs and the launch per phase
above 8,192 triangles, one and more levels of boxes above 1,024 positions (from
32,769), leaf sizes 1 to 255, equal codes throughout. The oracle's refit accepts
each layout and leaves every bound bit-identical (nothing is rounded, so there is
no tolerance)."""
import numpy as np
import pytest

from speedball_b200.scene import Mesh

from test_gpu_build import _check_layout, _gpu_build, ctx  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu


def _mesh(T, seed, equal=False):
    rng = np.random.default_rng(seed)
    c = np.zeros((T, 1, 3)) if equal else rng.uniform(-5, 5, (T, 1, 3))
    P = (c + rng.uniform(-0.1, 0.1, (T, 3, 3)) * (0 if equal else 1)).reshape(-1, 3).astype(np.float32)
    P[rng.random(P.shape) < 0.02] = -0.0  # both zeros as bounds
    return Mesh(P, rng.permutation(3 * T).astype(np.uint32).reshape(T, 3), np.zeros(T, np.uint32))


@pytest.mark.parametrize("T,leaf", [(8, 8), (9, 8), (31, 1), (32, 8), (33, 3), (255, 255), (300, 255), (1023, 8),
                                    (1024, 8), (1025, 1), (2048, 8), (2049, 8), (4097, 8), (8192, 8), (8193, 8),
                                    (32768, 8), (32769, 2), (70001, 8)])
def test_build_at_path_edges(ctx, T, leaf):  # noqa: F811
    lib, h = ctx
    m = _mesh(T, T)
    nodes, order = _gpu_build(lib, h, m, leaf)
    _check_layout(m, nodes, order, leaf)


@pytest.mark.parametrize("T", [40, 1500, 33000])
def test_build_with_equal_codes(ctx, T):  # noqa: F811
    lib, h = ctx
    m = _mesh(T, T, equal=True)
    nodes, order = _gpu_build(lib, h, m)
    assert np.array_equal(order, np.arange(T, dtype=np.uint32))  # ties keep their order
    _check_layout(m, nodes, order)
