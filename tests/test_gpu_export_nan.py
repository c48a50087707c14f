"""Surfaces with vertices that are no number (a field with NaN in it): a mesh of one component is
returned whole and as it is; beside others its volume compares with nothing, and none is kept."""
import numpy as np
import pytest
import torch

from anneal_gb300 import export as X
from anneal_gb300 import fem as G

pytestmark = pytest.mark.gpu


def _field(boxes):
    f = np.zeros((8, 10, 24), np.float32)   # indexed [k, j, i]
    for i0, i1 in boxes:
        f[2:6, 3:7, i0:i1] = 1.0
    f[4, 2, boxes[0][0] + 1] = np.nan   # beside the first box: its edges to it get no position
    return torch.as_tensor(f.ravel(), device="cuda")


def test_one_component_is_kept():
    f = _field([(3, 9)])
    grid = G.Grid((24, 10, 8), 0.5, (1.0, 2.0, 3.0))
    mc = X.MarchingCubes()
    mc.extract(f, grid.shape, 0.4, grid.h, grid.origin, 1)
    assert torch.unique(mc.components()).numel() == 1
    v, fc = (a.cpu().numpy() for a in mc.mesh_device())
    assert fc.shape[0] > 0 and not np.isfinite(v).all()
    dropped, volume = mc.prune(0.01)
    v2, fc2 = (a.cpu().numpy() for a in mc.mesh_device())
    assert dropped == 0 and np.isnan(volume)
    assert np.array_equal(v, v2, equal_nan=True) and np.array_equal(fc, fc2)
    mc.close()
    mesh = X.surface(grid, f, 0.4, upsample=1, smooth=0)
    assert np.array_equal(np.asarray(mesh.faces), fc)
    assert np.array_equal(np.asarray(mesh.vertices, np.float32), v, equal_nan=True)


def test_beside_others_none_is_kept():
    f = _field([(3, 9), (13, 19)])
    mc = X.MarchingCubes()
    mc.extract(f, (24, 10, 8), 0.4, 0.5, (1.0, 2.0, 3.0), 1)
    assert torch.unique(mc.components()).numel() == 2
    dropped, volume = mc.prune(0.01)
    assert dropped == 2 and volume == 0.0 and mc.nv == 0 and mc.nf == 0
    mc.close()
