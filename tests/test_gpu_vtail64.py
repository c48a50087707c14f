"""The FP64 cluster tail of the V-cycle against the same levels as separate launches: slabs along every
axis, odd and ragged sides, one layer to a CTA and several, grids whose whole V-cycle is the tail, and a
first level too large for it. The two V-cycles differ in the order of their sums only; the bars are those
of the FP32 comparison in the same ratio to the tolerance: 100 times it, of the largest displacement, and
CG iterations within 10 % (2 at least)."""
import numpy as np
import pytest

from anneal_gb300 import fem as G
from anneal_gb300 import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(8, 4, 4), (16, 8, 8), (7, 21, 6), (9, 7, 33), (33, 17, 9), (64, 32, 32), (61, 18, 37),
                                   (30, 62, 28), (18, 4, 70)])
def test_tail_matches_per_level_launches(monkeypatch, shape):
    w = P.cantilever(*shape)
    E = 1e-6 + P.random_density(shape, 3) ** 3
    out = {}
    for on in ("1", "0"):
        monkeypatch.setenv("ANL_TAIL", on)
        fem = G.FEM(G.Grid(w.shape, 1.0, (0, 0, 0)), w.active, w.fixed, 0.3, precision="fp64")
        u = fem.solve(fem.assemble(E[fem.act]), [fem.reduce_load(w.loads["c"])], rtol=1e-10)
        out[on] = u[0], fem.cg_iters[0]
        fem.close()
    (ut, it_t), (ul, it_l) = out["1"], out["0"]
    assert np.abs(ut - ul).max() <= 1e-8 * np.abs(ul).max()
    assert abs(it_t - it_l) <= max(2, it_l // 10), (it_t, it_l)
