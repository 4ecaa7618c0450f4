"""Which operators the FP64 contraction takes as digits: where digits below a
row's largest entry would lose entries that FP64 sums keep (banded, triangular,
diagonal, graded operators on graded data), the launch sums by FMAs and gives the
CUDA-core path's bits; the fast-diagonalisation factors keep their digits and are
held to the FMA path's error entry by entry."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from test_gpu_sliced_edges import randn, tp  # noqa: E402


def decay(n):
    return torch.exp(-torch.arange(n, dtype=torch.float64, device="cuda"))


def operators(n):
    from jaxfun_gb300.galerkin import DIRICHLET, FunctionSpace, Legendre, TensorProduct
    from jaxfun_gb300.la import poisson_tpmatrices

    D = FunctionSpace(n + 2, Legendre, bcs=DIRICHLET)
    A = poisson_tpmatrices(TensorProduct(D, D), 0.0)
    mass = A.tpmats[0].mats[1]
    i = np.arange(n)
    return {"identity": np.eye(n), "mass": np.asarray(mass),
            "triangular": np.where(i[None] > i[:, None], 2.0 * i[None], 0.0),
            "factor": A.lu_factor().W_host,
            "powers": np.linspace(-1.0, 1.0, n)[:, None] ** i[None]}


@pytest.mark.parametrize("n,B", [(62, 1001), (62, 61), (130, 40), (300, 5)])
@pytest.mark.parametrize("kind", ["identity", "mass", "triangular", "factor", "powers"])
def test_sparse_and_graded_operators_by_fma(n, B, kind):
    A = torch.as_tensor(np.ascontiguousarray(operators(n)[kind]), device="cuda")
    x = randn(5, B, n, n) * decay(n)[:, None] * decay(n)
    got, ref = tp([A, A], x), tp([A, A], x, cut=False)
    assert torch.equal(got, ref)
    if kind == "identity":
        assert torch.equal(got, x)
    # one such axis beside a dense one
    V = randn(6, n, n)
    got, ref = tp([A, V], x), tp([A, V], x, cut=False)
    mag = torch.einsum("ma,nb,iab->imn", A.abs(), V.abs(), x.abs())
    assert ((got - ref).abs() <= 4 * (2 * n + 2) * 2.0**-53 * mag).all()


def test_tpmatrix_entry_by_entry():
    from jaxfun_gb300.galerkin import DIRICHLET, FunctionSpace, Legendre, TensorProduct
    from jaxfun_gb300.la import poisson_tpmatrices

    n = 62
    D = FunctionSpace(n + 2, Legendre, bcs=DIRICHLET)
    for m in poisson_tpmatrices(TensorProduct(D, D), 0.0).tpmats:
        x = randn(7, 500, n, n) * decay(n)[:, None] * decay(n)
        a, b = (torch.as_tensor(np.ascontiguousarray(f), device="cuda") for f in m.mats)
        mag = torch.einsum("ma,nb,iab->imn", a.abs(), b.abs(), x.abs()) * abs(m.coefficient)
        one = torch.cat([m @ x[i:i + 1] for i in range(0, 500, 100)])  # small calls
        assert ((m @ x)[::100] - one).abs().le(4 * (2 * n + 3) * 2.0**-53 * mag[::100]).all()


@pytest.mark.parametrize("family", ["legendre", "chebyshev"])
def test_fast_diagonalisation_entry_by_entry(family):
    """rms error of each entry over the problems, against the FMA path's: the
    median below it, 99 % below 4 times it (rms of 12 samples on both sides:
    factors of up to 2 either way come from the samples alone)."""
    from jaxfun_gb300 import _lib
    from jaxfun_gb300.galerkin import DIRICHLET, Chebyshev, FunctionSpace, Legendre, TensorProduct
    from jaxfun_gb300.la import poisson_tpmatrices

    N, B = 128, 12
    D = FunctionSpace(N, Legendre if family == "legendre" else Chebyshev, bcs=DIRICHLET)
    T = TensorProduct(D, D)
    fac = poisson_tpmatrices(T, 0.0).lu_factor()
    n = fac.n
    k = (1.0 + torch.arange(N, dtype=torch.float64, device="cuda")) ** -2.0
    grid = TensorProduct(*([Legendre(N) if family == "legendre" else Chebyshev(N)] * 2))
    f = T.scalar_product(grid.backward(randn(8, B, N, N) * k[:, None] * k))
    E, W, lam = fac.device_factors()
    L = _lib.lib()
    out = []
    need = L.jfg_fd_solve_workspace_size(2, n, 64, 8)
    rhs = torch.cat([f] * 6)[:64].contiguous()
    for size in (need, need - 1):
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        u = torch.empty_like(rhs)
        st = L.jfg_fd_solve_f64(2, n, 64, E.data_ptr(), W.data_ptr(), lam.data_ptr(), None, None,
                                rhs.data_ptr(), u.data_ptr(), ws.data_ptr(), ws.numel(),
                                _lib.stream_handle())
        assert st == 0
        out.append(u[:B].cpu().numpy())
    ld = np.longdouble
    Eh, Wh, lh = (a.astype(ld) for a in (fac.E_host, fac.W_host, fac.lam_host))
    exact = np.stack([Wh @ ((Eh @ g.astype(ld) @ Eh.T) / (lh[:, None] + lh)) @ Wh.T
                      for g in f.cpu().numpy()])
    rms = [np.sqrt(((o - exact) ** 2).mean(0)).astype(float) for o in out]
    ratio = rms[0] / rms[1]
    assert not np.array_equal(out[0], out[1])  # digits on one side
    assert np.median(ratio) < 1.0 and np.quantile(ratio, 0.99) < 4.0


@pytest.mark.parametrize("n,B", [(62, 1001), (130, 40), (300, 8)])
def test_mantissas_near_two(n, B):
    """Rows whose largest entries have mantissas around 2 - 2^-6, from which their
    exponent counts one more, in both operands and signs."""
    near = torch.tensor([2.0 - 2.0**-52, 2.0 - 2.0**-6, 2.0 - 2.0**-6 - 2.0**-52, 2.0 - 2.0**-7,
                         1.0, 2.0 - 2.0**-5], dtype=torch.float64, device="cuda")
    g = torch.Generator(device="cuda")
    g.manual_seed(9)

    def pick(*shape):
        i = torch.randint(0, len(near), shape, device="cuda", generator=g)
        sign = torch.randint(0, 2, shape, device="cuda", generator=g) * 2.0 - 1.0
        return (near[i] * sign).double()

    A, V, x = pick(n, n), pick(n, n), pick(B, n, n)
    got, ref = tp([A, V], x), tp([A, V], x, cut=False)
    mag = torch.einsum("ma,nb,iab->imn", A.abs(), V.abs(), x.abs())
    assert ((got - ref).abs() <= 4 * (2 * n + 2) * 2.0**-53 * mag).all()


@pytest.mark.parametrize("K", [256, 257, 512])
def test_levels_past_their_exact_range(K):
    """K terms whose first three digits lie between 104 and 125: above 256 terms
    the FP32 sums of levels that count pass 2^24, on values of every parity, and
    the results are still those of FP64 sums."""
    g = torch.Generator(device="cuda")
    g.manual_seed(10)
    M, B = 130, 40

    def near(*shape):
        u = torch.rand(*shape, dtype=torch.float64, device="cuda", generator=g) - 0.5
        for _ in range(3):
            u = u / 256 + torch.randint(104, 126, shape, device="cuda", generator=g)
        return u * 2.0**-7

    I, A, x = near(16, 16), near(M, K), near(B, 16, K)
    got, ref = tp([I, A], x), tp([I, A], x, cut=False)
    mag = torch.einsum("ma,nb,iab->imn", I, A, x)
    assert ((got - ref).abs() <= 4 * (K + 16 + 2) * 2.0**-53 * mag).all()


@pytest.mark.parametrize("rows,cols,B,digits", [
    ((512,), (256,), 4, False), ((128,), (128,), 31, False), ((5,), (128,), 245, False),
    ((512, 512), (16, 16), 2, False), ((64, 64), (64, 64), 31, True),
    ((128, 128), (128, 128), 4, True), ((512,), (256,), 40, True)])
def test_calls_that_digits_would_slow_down(rows, cols, B, digits):
    """Room for digits is asked for where the passes save more than the cut costs."""
    from jaxfun_gb300 import _lib

    L = _lib.lib()
    a = len(rows), _lib.int_array(rows), _lib.int_array(cols), B, 8
    assert (L.jfg_tp_apply_workspace_size(*a) > L.jfg_tp_apply_fma_workspace_size(*a)) == digits
