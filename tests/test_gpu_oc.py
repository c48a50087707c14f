"""The OC update's multiplier search against the oracle's 36-step bisection: every filter halo, with and
without projection, tile edges, and targets that no multiplier reaches (the bisection then runs to
an end of its bracket). The bars are those of the oracle comparison of the kernels' tests: densities
within 1e-4, steps within 2."""
import numpy as np
import pytest
import torch

from anneal_gb300.context import Context, to_dev

pytestmark = pytest.mark.gpu
F32, U8 = torch.float32, torch.uint8


@pytest.mark.parametrize("shape", [(9, 4, 3), (33, 17, 9), (64, 8, 18)])
@pytest.mark.parametrize("r", [1.5, 2.6, 3.4, 4.5, 5.2])
@pytest.mark.parametrize("beta,share", [(0.0, 0.3), (1.0, 0.3), (4.0, 0.25), (0.0, 2.0), (2.0, 2.0), (0.0, 0.0), (2.0, 0.0)])
def test_multiplier_search_matches_oracle_bisection(oracle, shape, r, beta, share):
    rng = np.random.default_rng(int(10 * r) + shape[0])
    ne = int(np.prod(shape))
    active = rng.random(ne) > 0.15
    frozen = (rng.random(ne) < 0.05) & active
    phi = np.where(active, np.clip(rng.random(ne) + 0.3, 0, 1), 0.0).astype(np.float32)
    x = np.where(active, np.clip(rng.random(ne), 0.05, 1.0), 0.0).astype(np.float32)
    dcx = np.where(active, -np.exp(rng.normal(0, 2, ne)) * 1e-3, 0.0).astype(np.float32)
    dcx[rng.random(ne) < 0.05] = 0.0
    F = oracle.OracleFilter(shape, active, r)
    act = F.act
    dvx = np.zeros(ne, np.float32)
    dvx[act] = F.backward(phi[act].astype(float))
    vtarget = share * float(phi.sum())
    f64 = [a[act].astype(float) for a in (x, dcx, dvx, phi)]
    want, steps = oracle.oc_update(F, *f64, frozen[act], 0.2, beta, vtarget)
    c = Context(shape, 1.0, 0.3)
    c.set_domain(to_dev(active, U8), torch.zeros(c.ndof, dtype=U8, device="cuda"))
    c.filter_init(r)
    xn = torch.empty(ne, dtype=F32, device="cuda")
    got_steps, _ = c.oc_update(*(to_dev(a, F32) for a in (x, dcx, dvx, phi)), to_dev(frozen, U8), 0.2, beta, 0.5, vtarget,
                               xn)
    assert abs(got_steps - steps) <= 2
    assert np.abs(xn.cpu().numpy()[act] - want).max() < 1e-4
    c.close()
