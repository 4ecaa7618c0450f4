"""Edges of the FP64 contraction by digits: warps whose lanes take different
ways (rows past the last problem beside rows that are summed as they stand)."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def tp(mats, x, cut=True, out=None):
    """jfg_tp_apply_f64; with cut=False the workspace is one byte short of the
    room for digits, so that every pass runs on the CUDA cores."""
    from jaxfun_gb300 import _lib

    L = _lib.lib()
    rows, cols = [m.shape[0] for m in mats], [m.shape[1] for m in mats]
    r, c = _lib.int_array(rows), _lib.int_array(cols)
    need = L.jfg_tp_apply_workspace_size(len(mats), r, c, x.shape[0], 8)
    ws = torch.empty(need if cut else need - 1, dtype=torch.uint8, device="cuda")
    if out is None:
        out = torch.full([x.shape[0]] + rows, float("nan"), dtype=torch.float64, device="cuda")
    st = L.jfg_tp_apply_f64(len(mats), r, c, x.shape[0],
                            _lib.ptr_array([m.data_ptr() for m in mats]), x.data_ptr(),
                            out.data_ptr(), ws.data_ptr(), ws.numel(), _lib.stream_handle())
    assert st == 0, _lib.status_string(st)
    torch.cuda.synchronize()
    assert L.jfg_device_status() == 0
    return out


def randn(seed, *shape):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=g)


@pytest.mark.parametrize("B,K0,K1,M0,M1", [(1001, 49, 49, 51, 51), (3001, 17, 16, 31, 64),
                                           (131, 33, 63, 33, 129)])
def test_dead_and_special_rows_in_one_warp(B, K0, K1, M0, M1):
    """The last tile holds live rows, rows with infinities and NaNs and rows
    past the last problem, over several steps of columns: the same specials as
    the CUDA-core path, the other values of the live rows to the rounding of
    sums of K0 and K1 terms in either order of summation."""
    mats, x = [randn(1, M0, K0), randn(2, M1, K1)], randn(3, B, K0, K1)
    x[-1, -1, 3], x[-1, -3, 0], x[-2, -1, 1] = float("inf"), float("nan"), -float("inf")
    got, ref = tp(mats, x), tp(mats, x, cut=False)
    for kind in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(kind(got), kind(ref))
    mag = torch.einsum("ma,nb,iab->imn", mats[0].abs(), mats[1].abs(), x[:-2].abs())
    assert ((got[:-2] - ref[:-2]).abs() <= 8 * (K0 + K1 + 2) * 2.0**-52 * mag).all()
