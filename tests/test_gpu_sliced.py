"""The tensor-core FP64 contraction (operands cut into FP16 digits) against
extended-precision sums and the CUDA-core FP64 path, over the forms it takes:
edges of its tiles (32 or 16 rows of p, 128 operator rows, 64-element K
blocks, 16-element K steps), odd and aligned strides, operators of equal and
unequal axes, subsets, the three epilogues, and rows with infinities and NaNs."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _tp(mats, x, cut=True):
    """jfg_tp_apply_f64; with cut=False the workspace is one byte short of the
    room for digits, so that every pass runs on the CUDA cores."""
    from jaxfun_gb300 import _lib

    L = _lib.lib()
    nd = len(mats)
    rows, cols = [m.shape[0] for m in mats], [m.shape[1] for m in mats]
    B = x.shape[0]
    r, c = _lib.int_array(rows), _lib.int_array(cols)
    need = L.jfg_tp_apply_workspace_size(nd, r, c, B, 8)
    ws = torch.empty(need if cut else need - 1, dtype=torch.uint8, device="cuda")
    out = torch.full([B] + rows, float("nan"), dtype=torch.float64, device="cuda")
    st = L.jfg_tp_apply_f64(nd, r, c, B, _lib.ptr_array([m.data_ptr() for m in mats]),
                            x.data_ptr(), out.data_ptr(), ws.data_ptr(), ws.numel(),
                            _lib.stream_handle())
    assert st == 0, _lib.status_string(st)
    torch.cuda.synchronize()
    assert L.jfg_device_status() == 0
    return out


def _randn(seed, *shape):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=g)


# (batch, P, K, M): batch large enough for the tensor cores to be chosen
SHAPES = [
    (130, 33, 63, 31), (70, 64, 64, 64), (66, 31, 65, 129), (20, 97, 127, 128),
    (24, 62, 129, 66), (9, 100, 150, 148), (8, 96, 256, 200), (8, 45, 257, 130),
    (6, 40, 512, 130), (300, 16, 17, 257), (600, 17, 48, 33), (2, 33, 400, 513),
]


@pytest.mark.parametrize("B,P,K,M", SHAPES)
@pytest.mark.parametrize("scaled", [False, True])
def test_one_pass_against_extended_precision(B, P, K, M, scaled):
    """out = A x per row.  With c_k the operator's column exponents, a = A / c
    and y = x c, an operand keeps 61 bits below its row's maximum (twice K 2^-60
    of the product of the maxima), the digit products left out add at most
    7 K 2^-60, and the result is rounded once: within 2^-53 |ref| + K 2^-55
    max|a| max|y|.  The second axis' operator is the identity (one more rounding
    of the same kind, of rows whose maximum is the result's)."""
    A, x = _randn(1, M, K), _randn(2, B, P, K)
    if scaled:
        k = 1.0 + torch.arange(K, dtype=torch.float64, device="cuda")
        A, x = A * k**3, x * k**-5
    eye = torch.eye(P, dtype=torch.float64, device="cuda")
    out = _tp([eye, A], x)
    a, sel = A.cpu().numpy(), [0, B // 2, B - 1]
    y = x[sel].cpu().numpy()
    ref = np.einsum("mk,bpk->bpm", a.astype(np.longdouble), y.astype(np.longdouble))
    c = 2.0 ** np.floor(np.log2(np.abs(a).max(axis=0)))
    bound = np.abs(a / c).max(axis=1)[None, None, :] * np.abs(y * c).max(axis=2)[..., None]
    tol = (2.0**-53 * np.abs(ref) + K * 2.0**-55 * bound).astype(np.float64)
    second = 2.0**-53 * np.abs(ref) + P * 2.0**-55 * np.abs(ref).max(axis=1, keepdims=True)
    err = np.abs(out[sel].cpu().numpy() - ref)
    assert (err <= tol + second.astype(np.float64)).all(), float((err / (tol + second)).max())


def test_integers_are_exact_and_scales_do_not_matter():
    g = torch.Generator(device="cuda")
    g.manual_seed(5)

    def ints(*s):
        return torch.randint(-1000, 1000, s, device="cuda", generator=g).double()

    mats, x = [ints(53, 51), ints(51, 49)], ints(90, 51, 49)
    out = _tp(mats, x)
    assert torch.equal(out, _tp(mats, x, cut=False))
    for e in (-900, 900):
        assert torch.equal(_tp(mats, x * 2.0**e), out * 2.0**e)
    assert not _tp(mats, torch.zeros_like(x)).any()


def test_infinities_nans_and_scratch_limits():
    """Rows with specials, and results that leave the normal range, are those
    of the CUDA-core path: the same infinities and NaNs, the rest to FP64
    rounding of sums of K terms (K 2^-52 of the row's terms)."""
    B, K0, K1, M0, M1 = 90, 51, 49, 51, 53
    mats, x = [_randn(1, M0, K0), _randn(2, M1, K1)], _randn(3, B, K0, K1)
    x[3, 4, 5], x[7, 1, 2] = float("inf"), float("nan")
    x[9, 0, 0], x[9, 0, 1] = -float("inf"), float("inf")
    x[11] *= 1e307
    x[12] *= 2.0**-1060
    bad = mats[1].clone()
    bad[3, 3] = float("inf")
    for m in (mats, [mats[0], bad]):
        got, ref = _tp(m, x), _tp(m, x, cut=False)
        fin = torch.isfinite(got) & torch.isfinite(ref)
        same = (got == ref) | (got.isnan() & ref.isnan())
        # a sum may overflow on one side of the range's end and not on the other
        edge = (got.abs() > 1e307) | (ref.abs() > 1e307)
        assert (same | fin | edge).all()
        if m is mats:
            for b in (0, 50, 89):
                tol = (K0 + K1) * 2.0**-52 * (m[0].abs() @ x[b].abs() @ m[1].abs().T)
                assert ((got[b] - ref[b]).abs() <= tol).all()
            assert (got[12] - ref[12]).abs().max() <= 2.0**-1074 * K0 * K1 * 8


@pytest.mark.parametrize("ndim,n,batch", [(2, 62, 90), (2, 101, 40), (2, 254, 4), (3, 33, 20)])
def test_fast_diagonalisation(ndim, n, batch):
    """E, W passes and the eigenvalue divide: both FP64 paths agree to the
    rounding of 2 d sums of n terms, measured against the largest answer."""
    from jaxfun_gb300 import _lib

    L = _lib.lib()
    E, W = _randn(1, n, n) / n**0.5, _randn(2, n, n) / n**0.5
    lam = torch.linspace(1.0, 50.0, n, dtype=torch.float64, device="cuda")
    rhs = _randn(3, batch, *([n] * ndim))
    c0 = torch.linspace(0.5, 2.0, batch, dtype=torch.float64, device="cuda")
    c1 = torch.linspace(1.0, 3.0, batch, dtype=torch.float64, device="cuda")
    need = L.jfg_fd_solve_workspace_size(ndim, n, batch, 8)
    res = []
    for size in (need, need - 1):
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        out = torch.full_like(rhs, float("nan"))
        st = L.jfg_fd_solve_f64(ndim, n, batch, E.data_ptr(), W.data_ptr(), lam.data_ptr(),
                                c0.data_ptr(), c1.data_ptr(), rhs.data_ptr(), out.data_ptr(),
                                ws.data_ptr(), size, _lib.stream_handle())
        assert st == 0, _lib.status_string(st)
        res.append(out)
    torch.cuda.synchronize()
    assert L.jfg_device_status() == 0
    scale = res[1].abs().amax(dim=tuple(range(1, ndim + 1)), keepdim=True)
    assert ((res[0] - res[1]).abs() <= 2 * ndim * n * 2.0**-52 * scale).all()


@pytest.mark.parametrize("ndim,N,batch", [(2, 64, 40), (2, 131, 10), (3, 28, 30), (3, 33, 12)])
def test_variable_coefficient_operator(ndim, N, batch):
    """All passes of the operator (field multiply, accumulated outputs,
    operator segments) on both FP64 paths."""
    from jaxfun_gb300 import _lib
    from jaxfun_gb300.galerkin import DIRICHLET, FunctionSpace, Legendre, TensorProduct
    from jaxfun_gb300.la import VarCoefMatrix

    L = _lib.lib()
    D = FunctionSpace(N, Legendre, bcs=DIRICHLET)
    T = TensorProduct(*([D] * ndim))
    A = VarCoefMatrix(T, torch.exp(0.5 * _randn(4, batch, *([N] * ndim))))
    u = _randn(5, batch, *([N - 2] * ndim))
    need = L.jfg_varcoef_workspace_size(ndim, N - 2, N, batch, 8)
    res = []
    for size in (need, need - 1):
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        v = torch.full_like(u, float("nan"))
        st = L.jfg_varcoef_apply_f64(ndim, N - 2, N, batch, A.ops.data_ptr(), A.kw.data_ptr(),
                                     u.data_ptr(), v.data_ptr(), ws.data_ptr(), size,
                                     _lib.stream_handle())
        assert st == 0, _lib.status_string(st)
        res.append(v)
    torch.cuda.synchronize()
    assert L.jfg_device_status() == 0
    scale = res[1].abs().amax(dim=tuple(range(1, ndim + 1)), keepdim=True)
    assert ((res[0] - res[1]).abs() <= 2 * ndim * N * 2.0**-52 * scale).all()
