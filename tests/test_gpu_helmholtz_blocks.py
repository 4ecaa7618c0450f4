"""The Helmholtz row sweep around the line counts from which it goes through
shared-memory tiles and from which its blocks have eight warps instead of four:
the same bits as in small batches."""

import numpy as np
import pytest
import torch

from jaxfun_gb300.la.helmholtz import helmholtz_apply

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [2779, 2780, 4169, 4170, 5700])
def test_batches_around_the_change_of_block_size(batch):
    """Up to 256 and 384 lines per SM: 2779 and 4169 problems of 14 on 152 SMs."""
    N = 16
    rng = np.random.default_rng(3)
    u = torch.as_tensor(rng.standard_normal((batch, N - 2, N - 2)), device="cuda")
    a2 = rng.uniform(0.0, 100.0, batch)
    v = helmholtz_apply("legendre", N, a2, u)
    for i in [*range(0, batch, 499), batch - 7]:
        assert torch.equal(v[i:i + 7], helmholtz_apply("legendre", N, a2[i:i + 7], u[i:i + 7]))
