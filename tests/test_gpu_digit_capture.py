"""The FP64 contraction by digits under stream capture (transform and
fast-diagonalisation solve), and operators with infinities: equal specials, and
the finite entries to FP64 rounding."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from test_gpu_sliced_edges import randn, tp  # noqa: E402


@pytest.mark.parametrize("n,B", [(62, 1024), (126, 40)])
def test_captured_calls_give_the_same_bits(n, B):
    from jaxfun_gb300 import _lib

    L = _lib.lib()
    V, W = randn(1, n, n), randn(2, n, n)
    lam = randn(3, n).abs() + 1.0
    x = randn(4, B, n, n)
    y, u = torch.empty_like(x), torch.empty_like(x)
    size = _lib.int_array((n, n))
    mats = _lib.ptr_array([V.data_ptr(), W.data_ptr()])
    ws = torch.empty(max(L.jfg_tp_apply_workspace_size(2, size, size, B, 8),
                         L.jfg_fd_solve_workspace_size(2, n, B, 8)), dtype=torch.uint8,
                     device="cuda")

    def calls():
        s = _lib.stream_handle()
        assert L.jfg_tp_apply_f64(2, size, size, B, mats, x.data_ptr(), y.data_ptr(),
                                  ws.data_ptr(), ws.numel(), s) == 0
        assert L.jfg_fd_solve_f64(2, n, B, V.data_ptr(), W.data_ptr(), lam.data_ptr(), None, None,
                                  y.data_ptr(), u.data_ptr(), ws.data_ptr(), ws.numel(), s) == 0

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        calls()
    for seed in (5, 6):  # other inputs and another operator in the same buffers
        x.copy_(randn(seed, B, n, n))
        V.copy_(randn(seed + 10, n, n))
        graph.replay()
        got = y.clone(), u.clone()
        calls()
        torch.cuda.synchronize()
        assert torch.equal(got[0], y) and torch.equal(got[1], u)
    assert L.jfg_device_status() == 0


@pytest.mark.parametrize("B,n,m", [(1001, 49, 51), (40, 130, 129)])
def test_operator_with_infinities(B, n, m):
    """Rows 3 and 5 of the operator hold an infinity and a NaN: the same specials
    as the CUDA-core path, every other row's results to the rounding of sums of n
    terms in either order."""
    A, V, x = randn(1, m, n), randn(2, m, n), randn(3, B, n, n)
    A[3, 7], A[5, 0] = float("inf"), float("nan")
    got, ref = tp([A, V], x), tp([A, V], x, cut=False)
    for kind in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(kind(got), kind(ref))
    rows = [i for i in range(m) if i not in (3, 5)]
    mag = torch.einsum("ma,nb,iab->imn", A[rows].abs(), V.abs(), x.abs())
    assert ((got - ref)[:, rows].abs() <= 8 * (2 * n + 2) * 2.0**-52 * mag).all()
