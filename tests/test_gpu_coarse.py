"""The dense inverse of the coarsest grid (block Gauss-Jordan, 16 columns a step, 32 x 32 tiles).

On a grid that is its own coarsest level the V-cycle is that inverse, so CG has to finish at once:
an iteration leaves at most about eps * cond(K) of the residual (cond below 1e5 here), 6e-3 in
FP32 and 2e-11 in FP64, hence three iterations at most to 1e-6 and to 1e-10."""
import numpy as np
import pytest

from anneal_gb300 import fem as G
from anneal_gb300 import problems as P

pytestmark = pytest.mark.gpu


# unknowns 24, 54, 96, 144 (whole blocks and not, one tile and several), 180 and 360 (FP64 above
# 160), 648 (one element thick, the largest kind)
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 2, 1), (3, 3, 1), (3, 3, 2), (4, 3, 2), (5, 4, 3), (11, 8, 1)])
@pytest.mark.parametrize("precision,rtol", [("fp32", 1e-6), ("fp64", 1e-10)])
def test_coarsest_inverse_solves_at_once(shape, precision, rtol):
    w = P.cantilever(*shape)
    fem = G.FEM(G.Grid(w.shape, 1.0, (0, 0, 0)), w.active, w.fixed, 0.3, precision=precision)
    E = np.random.default_rng(sum(shape)).uniform(0.3, 1.0, w.nelem)
    K, F = fem.assemble(E), fem.reduce_load(w.loads["c"])
    u = fem.solve(K, [F], rtol=rtol)[0]
    assert fem.cg_iters[-1] <= 3
    assert np.linalg.norm(F - K @ u) <= 1.01 * rtol * np.linalg.norm(F)
    fem.close()
