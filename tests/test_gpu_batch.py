"""The K u passes of a batched solve share one wave of CTAs among the right-hand sides, in other
segments than a single solve's: sizes and slot counts where the segments are shortest and longest, do
not divide the columns, and one count above an eighth of the resident CTAs (a wave each). A node's
value does not depend on the segments, so every case is bit-identical to its own solve."""
import numpy as np
import pytest

from anneal_gb300 import fem as G
from anneal_gb300 import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,n", [((9, 5, 7), 3), ((31, 8, 16), 2), ((60, 14, 33), 5), ((61, 29, 31), 7),
                                     ((96, 48, 48), 2), ((29, 13, 12), 40)])
def test_batch_is_bit_identical_to_single_solves(shape, n):
    w = P.cantilever(*shape)
    E = 1e-6 + P.random_density(shape, 6) ** 3
    rng = np.random.default_rng(n)
    fem = G.FEM(G.Grid(shape, 1.0, (0, 0, 0)), w.active, w.fixed, 0.3, precision="fp32", multi="batch")
    es = fem.assemble(E[fem.act])
    loads = [fem.reduce_load(w.loads["c"] + 1e-3 * rng.normal(size=w.loads["c"].shape)) for _ in range(n)]
    together = fem.solve(es, loads, rtol=1e-6)
    its = list(fem.cg_iters)
    assert any(k[2] == n for k in fem._ctxs)  # one context with a slot per case
    for i in range(n):
        alone = fem.solve(es, [loads[i]], rtol=1e-6)
        assert np.array_equal(together[i], alone[0]), i
        assert its[i] == list(fem.cg_iters)[-1]
    fem.close()
