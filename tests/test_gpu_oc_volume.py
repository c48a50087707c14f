"""The volumes that decide the OC update's multiplier where they are no number."""
import numpy as np
import pytest
import torch

from anneal_gb300.context import Context, to_dev

pytestmark = pytest.mark.gpu
F32, U8 = torch.float32, torch.uint8


def _case(oracle, shape, r, seed):
    rng = np.random.default_rng(seed)
    ne = int(np.prod(shape))
    active = rng.random(ne) > 0.15
    frozen = (rng.random(ne) < 0.05) & active
    phi = np.where(active, np.clip(rng.random(ne) + 0.3, 0, 1), 0.0).astype(np.float32)
    x = np.where(active, np.clip(rng.random(ne), 0.05, 1.0), 0.0).astype(np.float32)
    dcx = np.where(active, -np.exp(rng.normal(0, 2, ne)) * 1e-3, 0.0).astype(np.float32)
    F = oracle.OracleFilter(shape, active, r)
    dvx = np.zeros(ne, np.float32)
    dvx[F.act] = F.backward(phi[F.act].astype(float))
    c = Context(shape, 1.0, 0.3)
    c.set_domain(to_dev(active, U8), torch.zeros(c.ndof, dtype=U8, device="cuda"))
    c.filter_init(r)
    return c, F, x, dcx, dvx, phi, frozen


# a volume that is no number is not above the target in the bisection, whatever the multiplier: it ends
# at the lower end of its bracket
@pytest.mark.parametrize("shape,r", [((9, 4, 3), 1.5), ((33, 17, 9), 2.6)])
@pytest.mark.parametrize("beta,bad", [(0.0, np.nan), (1.0, np.nan), (4.0, np.nan)])
def test_volume_that_is_no_number_ends_as_the_bisection(oracle, shape, r, beta, bad):
    c, F, x, dcx, dvx, phi, frozen = _case(oracle, shape, r, 5)
    design = np.flatnonzero(~frozen[F.act])
    phi[F.act[design[len(design) // 2]]] = bad
    f64 = [a[F.act].astype(float) for a in (x, dcx, dvx, phi)]
    vtarget = 0.3 * float(np.nansum(phi[np.isfinite(phi)]))
    want, steps = oracle.oc_update(F, *f64, frozen[F.act], 0.2, beta, vtarget)
    xn = torch.empty(c.ne, dtype=F32, device="cuda")
    got_steps, _ = c.oc_update(*(to_dev(a, F32) for a in (x, dcx, dvx, phi)), to_dev(frozen, U8), 0.2, beta, 0.5, vtarget,
                               xn)
    assert abs(got_steps - steps) <= 2
    assert np.abs(xn.cpu().numpy()[F.act] - want).max() < 1e-4
    c.close()
