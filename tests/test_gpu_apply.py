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


# grids on the two-kernel FP64 pass (a single element, partial warps and blocks, odd sides)
@pytest.mark.parametrize("shape", [(1, 1, 1), (5, 3, 2), (31, 9, 17), (64, 32, 32)])
def test_split_fp64_pass_matches_the_march(shape):
    """The FP64 pass of small levels against the marching one: a value is a sum of 8 corner forces of
    some 40 operations each, so the two orders differ by at most 8 * 40 * 1.1e-16 = 4e-14 of the
    forces' size, here bounded by the largest value of |K| |u|."""
    rng = np.random.default_rng(sum(shape))
    c = Context(shape, 1.0, 0.3, fp64=True)
    c.set_domain(torch.ones(c.ne, dtype=torch.uint8, device="cuda"), torch.zeros(c.ndof, dtype=torch.uint8, device="cuda"))
    E = to_dev(rng.uniform(0.1, 2.0, c.ne), torch.float32)
    u = to_dev(rng.normal(size=c.ndof), torch.float64)
    y, z = torch.empty_like(u), torch.empty_like(u)
    c.apply_K(E, u, y)
    c.profile_apply(u, z, 1)   # the solver's own pass on the same element scales
    bound = 2.0 * 8 * 4.0 * float(u.abs().max())   # E, corners, the row sums of |Ke| (below 4), u
    assert float((y - z).abs().max()) <= 4e-14 * bound
    c.close()
