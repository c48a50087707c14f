"""The removal of small components (anl_mc_prune) against the same steps in numpy: which components go,
the order of what is left, and its signed volume."""
import numpy as np
import pytest
import torch

from anneal_gb300 import export as X

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,fill,seed", [((5, 4, 3), 0.5, 0), ((16, 12, 10), 0.75, 1), ((40, 21, 17), 0.8, 2),
                                             ((30, 30, 30), 0.6, 3)])
@pytest.mark.parametrize("fraction", [0.0, 0.01, 0.6, 1.0])
def test_prune_matches_numpy(shape, fill, seed, fraction):
    rng = np.random.default_rng(seed)
    f = torch.as_tensor(rng.random(int(np.prod(shape))) * (rng.random(int(np.prod(shape))) > fill), dtype=torch.float32,
                        device="cuda")
    mc = X.MarchingCubes()
    mc.extract(f, shape, 0.3, 0.7, (3.0, -40.0, 0.25), 2)
    labels = mc.components().long().cpu().numpy()
    v, fc = (a.cpu().numpy() for a in mc.mesh_device())
    v, fc = v.astype(float), fc.astype(np.int64)
    uniq, comp = np.unique(labels, return_inverse=True)
    t = v[fc]
    tv = np.einsum("ij,ij->i", t[:, 0], np.cross(t[:, 1], t[:, 2])) / 6.0
    vols = np.abs(np.bincount(comp, weights=tv))
    keep = vols >= fraction * vols.max()
    want_v, want_f = v, fc
    if not keep.all():
        used, inv = np.unique(fc[keep[comp]].ravel(), return_inverse=True)
        want_v, want_f = v[used], inv.reshape(-1, 3)
    dropped, volume = mc.prune(fraction)
    got_v, got_f = (a.cpu().numpy() for a in mc.mesh_device())
    assert dropped == int((~keep).sum())
    assert np.array_equal(got_f, want_f) and np.array_equal(got_v.astype(float), want_v)
    # a face's volume is cut at 2^-60 of the bound 64^3 of a face, and numpy rounds each term
    assert abs(volume - tv[keep[comp]].sum()) <= 1e-12 * np.abs(tv).sum() + len(tv) * 64.0 ** 3 * 2.0 ** -60
    assert mc.prune(fraction)[0] == 0
    mc.close()
