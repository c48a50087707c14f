"""The cluster tail of the V-cycle against the same levels as separate launches: slabs along every
axis, odd and ragged sides, one layer to a CTA and several, more CTAs than layers, grids whose whole
V-cycle is the tail, and slots of a batch. The two V-cycles differ in the order of their sums, so the bars
are those of the existing comparison: 1e-6 of the largest displacement at a tolerance of 1e-8, and CG
iterations within 10 % (2 at least)."""
import numpy as np
import pytest

from anneal_gb300 import fem as G
from anneal_gb300 import problems as P

pytestmark = pytest.mark.gpu


def _solve(w, E, loads, **kw):
    fem = G.FEM(G.Grid(w.shape, 1.0, (0, 0, 0)), w.active, w.fixed, 0.3, precision="fp32", **kw)
    u = fem.solve(fem.assemble(E[fem.act]), [fem.reduce_load(F) for F in loads], rtol=1e-8)
    its = list(fem.cg_iters)
    fem.close()
    return u, its


@pytest.mark.parametrize("shape", [(16, 8, 8), (7, 21, 6), (9, 7, 33), (33, 17, 9), (64, 32, 32), (61, 18, 37), (30, 62, 28),
                                   (18, 4, 70)])
def test_tail_matches_per_level_launches(monkeypatch, shape):
    w = P.cantilever(*shape)
    E = 1e-6 + P.random_density(shape, 3) ** 3
    out = {}
    for on in ("1", "0"):
        monkeypatch.setenv("ANL_TAIL", on)
        out[on] = _solve(w, E, [w.loads["c"]])
    (ut, it_t), (ul, it_l) = out["1"], out["0"]
    assert np.abs(ut[0] - ul[0]).max() <= 1e-6 * np.abs(ul[0]).max()
    assert abs(it_t[0] - it_l[0]) <= max(2, it_l[0] // 10), (it_t, it_l)


def test_tail_slots_are_bit_identical_to_single_solves():
    w = P.cantilever(33, 17, 9)
    E = 1e-6 + P.random_density(w.shape, 4) ** 3
    rng = np.random.default_rng(2)
    loads = [w.loads["c"], rng.normal(size=w.ndof), rng.normal(size=w.ndof)]
    together, its = _solve(w, E, loads, multi="batch")
    for k, F in enumerate(loads):
        alone, it = _solve(w, E, [F])
        assert np.array_equal(together[k], alone[0]) and its[k] == it[0]
