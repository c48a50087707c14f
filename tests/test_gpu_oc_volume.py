"""The volumes that decide the OC update's multiplier: their precision, and values that are no number."""
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
# at the lower end of its bracket; an infinite one is above it, and it ends at the upper end. (With no
# projection an infinite phi is no number either: the filter's zero weights meet it.)
@pytest.mark.parametrize("shape,r", [((9, 4, 3), 1.5), ((33, 17, 9), 2.6), ((33, 17, 9), 3.4)])
@pytest.mark.parametrize("beta,bad", [(0.0, np.nan), (1.0, np.nan), (4.0, np.nan), (1.0, np.inf), (4.0, np.inf)])
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


@pytest.mark.parametrize("r", [1.5, 2.6, 3.4])
def test_projected_volume_is_summed_in_double_precision(r):
    """One design element beside many frozen ones, whose phi add up to 2^17.6 and are multiples of
    2^-34: FP64 holds their sum exactly in any order. The target leaves the design element, of phi
    2^-14, an xp of 0.55. FP64 rounds where that element's share is added: at most 2^-36 at the last
    sums, half as much where two halves meet and so on, 2^-35 in all and 2^-36 in the target, 2^-20.4 of
    the element's phi; the projection and the multiplier in FP32 add 8 units of 2^-24. Sums of float
    pairs (48 bits of 2^17.6, 2^-16 of that phi) miss the bar of 2^-19."""
    shape = (64, 64, 32)
    ne = int(np.prod(shape))
    rng = np.random.default_rng(8)
    big = rng.integers(2 ** 23, 2 ** 24, ne) * 2.0 ** -23
    small = rng.integers(2 ** 23, 2 ** 24, ne) * 2.0 ** -34
    phi = np.where(rng.random(ne) < 0.5, big, small).reshape(32, 64, 64)   # indexed [k, j, i]
    active = np.ones(phi.shape, bool)
    active[7:18, 21:32, 35:46] = False   # nothing within the filter's reach of the design element
    active[12, 26, 40] = True
    frozen = active.copy()
    frozen[12, 26, 40] = False
    phi[~active] = 0.0
    phi[12, 26, 40] = 2.0 ** -14
    assert np.array_equal(phi, phi.astype(np.float32))
    units = np.rint(phi[frozen] * 2.0 ** 34).astype(np.int64)
    vtarget = float(int(units.sum()) * 2.0 ** -34 + 0.55 * 2.0 ** -14)
    c = Context(shape, 1.0, 0.3)
    c.set_domain(to_dev(active.ravel(), U8), torch.zeros(c.ndof, dtype=U8, device="cuda"))
    c.filter_init(r)
    x = np.where(frozen, 1.0, np.where(active, 0.5, 0.0)).ravel()
    dcx, dvx = np.where(active & ~frozen, -1.0, 0.0).ravel(), np.where(active & ~frozen, 1.0, 0.0).ravel()
    frz = to_dev(frozen.ravel(), U8)
    xn, xp = (torch.empty(ne, dtype=F32, device="cuda") for _ in range(2))
    c.oc_update(*(to_dev(a, F32) for a in (x, dcx, dvx, phi.ravel())), frz, 0.2, 1.0, 0.5, vtarget, xn)
    c.physical(xn, frz, 1.0, 0.5, xp)
    got = float(xp.reshape(32, 64, 64)[12, 26, 40])
    assert abs(got - 0.55) <= 2.0 ** -19
    c.close()
