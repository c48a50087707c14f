"""K u through the caller's entry point, which masks u and forms the element scale on the way: against
itself with y in u's place (that call copies u first), on tile and segment edges. Both take the same
products in the same order, so they agree bit for bit."""
import numpy as np
import pytest
import torch

from anneal_gb300.context import Context, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (29, 14, 3), (30, 15, 8), (31, 7, 40), (62, 33, 17)])
@pytest.mark.parametrize("fp64", [False, True])
def test_fused_apply_matches_in_place_apply(shape, fp64):
    rng = np.random.default_rng(sum(shape))
    c = Context(shape, 0.7, 0.3, fp64=fp64)
    active = rng.random(c.ne) > 0.2
    active[0] = True
    fixed = rng.random(c.ndof) < 0.1
    c.set_domain(to_dev(active, torch.uint8), to_dev(fixed, torch.uint8))
    E = to_dev(rng.uniform(0.1, 2.0, c.ne), torch.float32)   # non-zero on inactive elements too
    u = to_dev(rng.normal(size=c.ndof), c.vdtype)            # non-zero on fixed unknowns too
    y = torch.empty_like(u)
    c.apply_K(E, u, y)
    c.apply_K(E, u, u)
    assert torch.equal(y, u)
    c.close()
