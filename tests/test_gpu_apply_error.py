"""The rounding error of the caller's FP32 K u on a smooth displacement field, where the forces of
neighbouring elements nearly cancel. The bars are what corner forces added one by one give for the same
inputs (1.2717e-7 and 1.3578e-7 of the result, root mean square), rounded up in the fourth digit."""
import numpy as np
import pytest
import torch

from anneal_gb300.context import Context, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,bar", [((61, 33, 29), 1.272e-7), ((97, 53, 34), 1.358e-7)])
def test_rounding_error_on_a_smooth_field(shape, bar):
    nx, ny, nz = shape
    k, j, i = np.meshgrid(*(np.arange(n + 1) / n for n in (nz, ny, nx)), indexing="ij")
    u = np.stack([np.sin(2 * i + j) * k, np.cos(3 * i - k) + j * j, i * i * j], -1).ravel()
    c, d = Context(shape, 0.7, 0.3), Context(shape, 0.7, 0.3, fp64=True)
    for x in (c, d):
        x.set_domain(torch.ones(c.ne, dtype=torch.uint8, device="cuda"),
                     torch.zeros(c.ndof, dtype=torch.uint8, device="cuda"))
    E = to_dev(np.random.default_rng(7).uniform(0.05, 1.0, c.ne), torch.float32)
    u = to_dev(u, torch.float32)
    y, z = torch.empty_like(u), torch.empty(c.ndof, dtype=torch.float64, device="cuda")
    c.apply_K(E, u, y)
    d.apply_K(E, u.double(), z)
    assert float((y - z).norm() / z.norm()) <= bar
    c.close()
    d.close()
