"""The Helmholtz row sweep at the edges of its tiles (32 lines per warp, 16
columns per step): line counts and lengths around them, against the oracle's
dense matrices, and uneven batches whose lines of different length share a
warp."""

import numpy as np
import pytest
import torch

from jaxfun_gb300.la.helmholtz import UnevenHelmholtzSolver, helmholtz_apply
from oracle import spectral as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family", ["legendre", "chebyshev"])
@pytest.mark.parametrize("N,batch", [(3, 5), (4, 40), (16, 3), (17, 2), (18, 19), (33, 1),
                                     (34, 9), (50, 11), (131, 2)])
def test_apply_matches_dense(family, N, batch):
    """Sums of at most N terms of the dense product's size: N^2 2^-52 of the
    largest entry of |A| |u|."""
    Vo = O.Space1D(family, N, True)
    K, M = Vo.stiffness_matrix(), Vo.mass_matrix()
    rng = np.random.default_rng(N)
    u = rng.standard_normal((batch, N - 2, N - 2))
    a2 = rng.uniform(0.0, 100.0, batch)
    v = helmholtz_apply(family, N, a2, u).cpu().numpy()
    for b in range(batch):
        terms = [(a2[b], [M, M]), (1.0, [K, M]), (1.0, [M, K])]
        ref = O.tp_apply(terms, u[b])
        size = O.tp_apply([(c, [abs(m) for m in ms]) for c, ms in terms], abs(u[b])).max()
        assert np.abs(v[b] - ref).max() <= N * N * 2.0**-52 * size


@pytest.mark.parametrize("family", ["legendre", "chebyshev"])
def test_lines_of_different_length_in_one_warp(family):
    """Small sizes, one or two problems each, so that a warp's 32 lines belong
    to several problems: residuals of the packed solve against dense algebra
    at the solve's tolerance."""
    Ns = np.array([4, 5, 6, 7, 9, 12, 17, 18, 20, 35, 36, 67])
    rng = np.random.default_rng(1)
    alphas = rng.uniform(0.5, 30.0, len(Ns))
    rhs = [rng.standard_normal((N - 2, N - 2)) for N in Ns]
    S = UnevenHelmholtzSolver(family, Ns, alphas)
    with torch.cuda.stream(torch.cuda.Stream()):
        xs, _ = S.solve(rhs, tol=1e-12)
    torch.cuda.synchronize()
    for b, N in enumerate(Ns):
        Vo = O.Space1D(family, int(N), True)
        K, M = Vo.stiffness_matrix(), Vo.mass_matrix()
        x = xs[b].cpu().numpy()
        terms = [(alphas[b] ** 2, [M, M]), (1.0, [K, M]), (1.0, [M, K])]
        r = rhs[b] - O.tp_apply(terms, x)
        size = O.tp_apply([(c, [abs(m) for m in ms]) for c, ms in terms], abs(x)).max()
        assert np.linalg.norm(r) <= 1e-12 * np.linalg.norm(rhs[b]) + N * N * 2.0**-52 * size
