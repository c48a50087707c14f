"""A filter set up on one stream and used on another."""
import numpy as np
import pytest
import torch

from anneal_gb300.context import Context, to_dev

pytestmark = pytest.mark.gpu


def test_filter_init_is_complete_on_return():
    shape = (40, 24, 16)
    rng = np.random.default_rng(0)
    c = Context(shape, 1.0, 0.3)
    c.set_domain(to_dev(rng.random(c.ne) > 0.2, torch.uint8), torch.zeros(c.ndof, dtype=torch.uint8, device="cuda"))
    x = to_dev(rng.random(c.ne), torch.float32)
    want, got = torch.empty_like(x), torch.empty_like(x)
    c.filter_init(2.6)
    c.filter_fwd(x, want)
    c.filter_init(1.5)   # another Hs, so that the next one has to be written again
    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        torch.cuda._sleep(200_000_000)   # about 0.1 s of work ahead of the filter's
        c.filter_init(2.6)
        assert a.query()
    with torch.cuda.stream(b):
        c.filter_fwd(x, got)
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    c.close()
