"""The density filter at every halo (R = 1..5) and at the edges of its tiles (32 x 8 columns, chunks
of 4 to 16 layers), against a plain FP64 convolution.

A value is a sum of positive terms rounded at most 8 (class sum) + 21 (classes) + 11 (layers) + 1
times, its normalisation Hs as often, and divided once: at most 83 roundings of 6e-8, 5e-6."""
import numpy as np
import pytest
import torch
from scipy.ndimage import convolve

from anneal_gb300.context import Context, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 3, 2), (32, 8, 16), (33, 9, 17), (70, 17, 41)])
@pytest.mark.parametrize("r", [1.0, 1.5, 2.0, 2.5, 3.0, 3.6, 4.5, 5.9])
def test_filter_matches_plain_convolution(shape, r):
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + int(10 * r))
    act = rng.random((nz, ny, nx)) > 0.2
    v = rng.uniform(0.1, 1.0, (nz, ny, nx))
    R = max(int(np.ceil(r)) - 1, 1)
    k = np.maximum(0.0, r - np.sqrt(sum(a ** 2 for a in np.meshgrid(*[np.arange(-R, R + 1)] * 3, indexing="ij"))))
    hs = convolve(act.astype(float), k, mode="constant")
    hs[hs == 0] = 1.0
    want_f = convolve(v * act, k, mode="constant") / hs * act
    want_b = convolve(v * act / hs, k, mode="constant") * act
    c = Context(shape, 1.0, 0.3)
    c.set_domain(to_dev(act.ravel(), torch.uint8), torch.zeros(c.ndof, dtype=torch.uint8, device="cuda"))
    c.filter_init(r)
    out = torch.empty(c.ne, dtype=torch.float32, device="cuda")
    for fn, want in ((c.filter_fwd, want_f), (c.filter_bwd, want_b)):
        fn(to_dev(v.ravel(), torch.float32), out)
        got = out.cpu().numpy().reshape(nz, ny, nx)
        assert np.abs(got - want).max() <= 5e-6 * np.abs(want).max()
    c.close()
