"""FP64 contraction by digits for operators of up to 64 x 64 (input rows as the
MMA's M operand), at the edges of its tiles: 128 rows flattened over the
problems, operator halves of 32 rows, 16-element K steps, odd strides, the
divide epilogue, rows with infinities and NaNs."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _tp(mats, x, cut=True):
    from jaxfun_gb300 import _lib

    L = _lib.lib()
    rows, cols = [m.shape[0] for m in mats], [m.shape[1] for m in mats]
    r, c = _lib.int_array(rows), _lib.int_array(cols)
    need = L.jfg_tp_apply_workspace_size(len(mats), r, c, x.shape[0], 8)
    ws = torch.empty(need if cut else need - 1, dtype=torch.uint8, device="cuda")
    out = torch.full([x.shape[0]] + rows, float("nan"), dtype=torch.float64, device="cuda")
    st = L.jfg_tp_apply_f64(len(mats), r, c, x.shape[0],
                            _lib.ptr_array([m.data_ptr() for m in mats]), x.data_ptr(),
                            out.data_ptr(), ws.data_ptr(), ws.numel(), _lib.stream_handle())
    assert st == 0, _lib.status_string(st)
    torch.cuda.synchronize()
    assert L.jfg_device_status() == 0
    return out


@pytest.mark.parametrize("B,K0,K1,M0,M1", [
    (1000, 62, 62, 64, 64), (997, 64, 63, 33, 32), (700, 49, 51, 51, 49), (3001, 17, 16, 31, 64),
    (5000, 15, 33, 48, 16), (9000, 8, 48, 9, 1), (400, 64, 64, 64, 64), (40000, 3, 64, 5, 63),
])
def test_two_passes_against_cuda_cores(B, K0, K1, M0, M1):
    """Same sums as the CUDA-core path to FP64 rounding: a pass is within K 2^-52
    of the sum of its terms' magnitudes on either side (the digits' own error is
    below that of the running sum), two passes within (K0 + K1 + 2) 2^-52 of the
    product with magnitudes throughout, which the digits' row-wise scales can
    exceed by the ratio of a row's largest to its mean: factor 8."""
    g = torch.Generator(device="cuda")
    g.manual_seed(B + K0)
    mats = [torch.randn(m, k, dtype=torch.float64, device="cuda", generator=g)
            for m, k in ((M0, K0), (M1, K1))]
    x = torch.randn(B, K0, K1, dtype=torch.float64, device="cuda", generator=g)
    got, ref = _tp(mats, x), _tp(mats, x, cut=False)
    mag = torch.einsum("ma,nb,iab->imn", mats[0].abs(), mats[1].abs(), x.abs())
    assert ((got - ref).abs() <= 8 * (K0 + K1 + 2) * 2.0**-52 * mag).all()
    # integers below the digits' width are exact on either path
    ints = [torch.round(8 * m) for m in mats]
    xi = torch.round(8 * x)
    assert torch.equal(_tp(ints, xi), _tp(ints, xi, cut=False))


def test_specials_stay_in_their_rows():
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    mats = [torch.randn(51, 49, dtype=torch.float64, device="cuda", generator=g) for _ in range(2)]
    x = torch.randn(1000, 49, 49, dtype=torch.float64, device="cuda", generator=g)
    x[3, 4, 5], x[127, 1, 2] = float("inf"), float("nan")
    x[128, 0, 0], x[128, 0, 1] = -float("inf"), float("inf")
    x[500] = 0.0
    x[600] *= 2.0**-1060
    got, ref = _tp(mats, x), _tp(mats, x, cut=False)
    for bad in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(bad(got), bad(ref))
    assert not got[500].any()
    assert torch.isfinite(got[[0, 2, 4, 126, 129, 600]]).all()


@pytest.mark.parametrize("B,n", [(700, 62), (2500, 17)])
def test_divide_epilogue_with_problem_shifts(B, n):
    """Fast diagonalisation with a shift per problem, digits against CUDA cores:
    four passes and a division, each to FP64 rounding of the magnitudes."""
    from jaxfun_gb300 import _lib

    L = _lib.lib()
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    e, w = (torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g) for _ in range(2))
    lam = 1.0 + torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    c0, c1 = (0.5 + torch.rand(B, dtype=torch.float64, device="cuda", generator=g)
              for _ in range(2))
    x = torch.randn(B, n, n, dtype=torch.float64, device="cuda", generator=g)
    need = L.jfg_fd_solve_workspace_size(2, n, B, 8)
    res = []
    for size in (need, need - 1):
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        out = torch.full_like(x, float("nan"))
        st = L.jfg_fd_solve_f64(2, n, B, e.data_ptr(), w.data_ptr(), lam.data_ptr(),
                                c0.data_ptr(), c1.data_ptr(), x.data_ptr(), out.data_ptr(),
                                ws.data_ptr(), ws.numel(), _lib.stream_handle())
        assert st == 0, _lib.status_string(st)
        torch.cuda.synchronize()
        assert L.jfg_device_status() == 0
        res.append(out)
    den = c0[:, None, None] + c1[:, None, None] * (lam[:, None] + lam[None, :])
    mag = torch.einsum("ma,nb,iab->imn", e.abs(), e.abs(), x.abs()) / den
    mag = torch.einsum("ma,nb,iab->imn", w.abs(), w.abs(), mag)
    assert ((res[0] - res[1]).abs() <= 8 * (4 * n + 5) * 2.0**-52 * mag).all()
