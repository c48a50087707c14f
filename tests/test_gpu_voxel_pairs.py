"""The voxeliser's pair lists, quotients from reciprocals and element stacks at the sizes where they can
go wrong, bit for bit against the oracle: triangles with many thousand columns and with none (their
offsets in shared memory or not), determinants of zero and beyond the reciprocals' range, every stack
height and heights that leave a partial stack, and one column of elements."""
import numpy as np
import pytest

from anneal_gb300 import geometry as G
from anneal_gb300.fem import Grid
from oracle import voxel_oracle as VO

pytestmark = pytest.mark.gpu


def _same(tri, shape, h, origin, s):
    g = Grid(shape, h, origin)
    assert np.array_equal(G.voxel_fill(tri, g, s=s), VO.voxel_fill(tri, g.shape, g.h, g.origin, s))


@pytest.mark.parametrize("s", [1, 2, 3, 5, 8, 9, 11, 16])
@pytest.mark.parametrize("shape", [(7, 5, 3), (4, 9, 13), (1, 1, 22)])
def test_stacks(shape, s):
    V, F = G.icosphere(3, 0.46, (0.5, 0.5, 0.5))
    _same((V * np.array(shape, float))[F], shape, 1.0, (0.0, 0.0, 0.0), s)


@pytest.mark.parametrize("shape,s", [((90, 70, 20), 3), ((160, 3, 9), 4)])
def test_few_large_triangles(shape, s):
    rot = np.linalg.qr(np.random.default_rng(5).normal(size=(3, 3)))[0]
    V, F = G.box(tuple(0.5 * n for n in shape), tuple(0.5 * n for n in shape), rot)
    _same(V[F], shape, 1.0, (0.0, 0.0, 0.0), s)


@pytest.mark.parametrize("sub,s", [(6, 1), (6, 2)])
def test_triangles_finer_than_the_columns(sub, s):
    """20 4^6 triangles over few columns: most have no column, so a block's pairs span more triangles
    than its shared memory holds."""
    V, F = G.icosphere(sub, 2.9, (3.0, 3.1, 3.2))
    big, Fb = G.box((30.0, 30.0, 2.0), (15.0, 15.0, 10.0), np.eye(3))
    _same(np.concatenate([V[F], big[Fb]]), (30, 30, 12), 1.0, (0.0, 0.0, 0.0), s)


@pytest.mark.parametrize("scale", [2.0 ** -300, 2.0 ** -190, 2.0 ** 150, 2.0 ** 250, 1e7])
def test_scales(scale):
    V, F = G.icosphere(3, 5.0, (6.0, 6.1, 6.2))
    _same(V[F] * scale, (12, 12, 12), scale, (0.0, 0.0, 0.0), 3)


def test_degenerate_triangles_add_nothing():
    rng = np.random.default_rng(8)
    V, F = G.icosphere(3, 5.0, (6.0, 6.1, 6.2))
    a, b = rng.uniform(1, 11, (2, 300, 3))
    flat = np.stack([a, b, a], 1)                       # a determinant of exactly zero
    thin = np.stack([a, b, 0.5 * (a + b)], 1)           # and of rounding size
    up = np.stack([a, a + [0, 0, 3.0], b], 1)
    _same(np.concatenate([V[F], flat, up, thin]), (12, 12, 12), 1.0, (0.0, 0.0, 0.0), 3)
