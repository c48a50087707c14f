"""A halo wait of the cluster tail that runs out fails the solve, whichever thread waited. The waits are
only counted as run out here (ANL_TAIL_LOSE_FROM, in the first CTA's threads from that one on): on
16 x 16 x 16 a CTA computes two layers of 256 elements, one to a thread, and but for the last owns one
plane of 17 x 17 nodes, so its threads from 289 on can wait for a halo plane and own no node."""
import numpy as np
import pytest
import torch

from anneal_gb300 import _native as N
from anneal_gb300 import problems as P
from anneal_gb300.context import Context, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lose_from,fails", [(None, False), (0, True), (200, True), (300, True), (512, False)])
def test_lost_halo_fails_the_solve(monkeypatch, lose_from, fails):
    if lose_from is not None:
        monkeypatch.setenv("ANL_TAIL_LOSE_FROM", str(lose_from))
    w = P.cantilever(16, 16, 16)
    c = Context(w.shape, 1.0, 0.3)
    fixed = np.zeros(c.ndof, np.uint8)
    fixed[np.asarray(w.fixed, np.int64)] = 1
    c.set_domain(to_dev(w.active, torch.uint8), to_dev(fixed, torch.uint8))
    F = to_dev(np.where(fixed, 0.0, w.loads["c"])[None], torch.float64)
    st, _, _ = c.solve(torch.ones(c.ne, device="cuda"), F, torch.zeros_like(F), 1e-6)
    assert st == (N.ANL_ERR_NONFINITE if fails else N.ANL_OK)
    c.close()
