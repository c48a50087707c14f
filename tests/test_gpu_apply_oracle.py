"""The caller's K u against the FP64 oracle where the pass has something to mask: an h other than 1,
element scales on inactive elements and values on fixed unknowns, on tile and segment edges; then with y
in u's place, with y over the element scales (which takes the separate passes), and the element scales that
the call leaves for the next pass. The bars are those of the kernels' oracle comparison (E is rounded to
FP32 on input: 1e-6 of the largest value in FP64, 2e-6 in FP32)."""
import numpy as np
import pytest
import torch

from anneal_gb300.context import Context, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (29, 14, 3), (31, 7, 40), (62, 33, 17)])
@pytest.mark.parametrize("fp64", [False, True])
def test_apply_matches_oracle_through_every_route(oracle, shape, fp64):
    rng = np.random.default_rng(sum(shape))
    ne, ndof = int(np.prod(shape)), 3 * int(np.prod([s + 1 for s in shape]))
    active = rng.random(ne) > 0.2
    active[0] = True
    fixed = rng.random(ndof) < 0.1
    E = rng.uniform(0.1, 2.0, ne).astype(np.float32)
    u = rng.normal(size=ndof).astype(np.float32)
    fem = oracle.OracleFEM(shape, 0.7, active, np.flatnonzero(fixed), 0.3)
    want = fem.apply(E[fem.act].astype(float), np.where(fem.mask, u, 0.0))
    bar = (1e-6 if fp64 else 2e-6) * np.abs(want).max()
    c = Context(shape, 0.7, 0.3, fp64=fp64)
    c.set_domain(to_dev(active, torch.uint8), to_dev(fixed, torch.uint8))
    Ed, ud = to_dev(E, torch.float32), to_dev(u, c.vdtype)

    def check(y):
        assert np.abs(y.cpu().numpy().astype(float) - want).max() <= bar

    y = torch.empty_like(ud)
    c.apply_K(Ed, ud, y)
    check(y)
    z = ud * to_dev(fem.mask, c.vdtype)
    c.profile_apply(z, y, 1)     # the element scales that the call stored
    check(y)
    z = ud.clone()
    c.apply_K(Ed, z, z)
    check(z)
    over = torch.zeros(ndof, dtype=c.vdtype, device="cuda")
    inside = over.view(torch.float32)[:ne]
    inside.copy_(Ed)
    c.apply_K(inside, ud, over)
    check(over)
    c.close()
