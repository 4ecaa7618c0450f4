"""Channel mixing of the spectral neural operator, forward and backward, against
FP64 sums: batches and modes around the kernels' steps (32 samples, one or four
modes a block), channel counts with and without 16-byte rows."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _randn(seed, *shape):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(*shape, device="cuda", generator=g)


@pytest.mark.parametrize("B,Q,C", [(1, 8, 1), (32, 1024, 64), (33, 512, 64), (70, 520, 20),
                                   (5, 24, 3), (64, 1032, 37), (300, 64, 64)])
def test_forward(B, Q, C):
    """FP32 sums of C terms (C 2^-23 of their magnitudes), rounded to BF16 (2^-8)."""
    from jaxfun_gb300 import _lib

    R, x = _randn(1, Q, C, C), _randn(2, B, Q, C)
    out = torch.full((B, C, Q), float("nan"), dtype=torch.bfloat16, device="cuda")
    _lib.check(_lib.lib().jfg_sno_modemix_fwd(B, Q, C, R.data_ptr(), x.data_ptr(), out.data_ptr(),
                                              _lib.stream_handle()), "fwd")
    ref = torch.einsum("qoi,bqi->boq", R.double(), x.double())
    mag = torch.einsum("qoi,bqi->boq", R.double().abs(), x.double().abs())
    tol = 2.0**-8 * ref.abs() + (C + 1) * 2.0**-23 * mag
    assert ((out.double() - ref).abs() <= tol).all()


@pytest.mark.parametrize("B,Q,C", [(1, 1, 1), (32, 1024, 64), (33, 515, 64), (70, 516, 20),
                                   (7, 13, 5), (65, 600, 37), (300, 30, 64), (0, 8, 16)])
def test_backward(B, Q, C):
    """As above; dR is the FP32 sum over B samples."""
    from jaxfun_gb300 import _lib

    R, x, dy = _randn(1, Q, C, C), _randn(2, B, Q, C), _randn(3, B, Q, C)
    dx = torch.full((B, C, Q), float("nan"), dtype=torch.bfloat16, device="cuda")
    dR = torch.full((Q, C, C), float("nan"), device="cuda")
    _lib.check(_lib.lib().jfg_sno_modemix_bwd(B, Q, C, R.data_ptr(), x.data_ptr() or R.data_ptr(),
                                              dy.data_ptr() or R.data_ptr(),
                                              dx.data_ptr() or R.data_ptr(), dR.data_ptr(),
                                              _lib.stream_handle()), "bwd")
    R64, x64, d64 = R.double(), x.double(), dy.double()
    ref = torch.einsum("qoi,bqo->biq", R64, d64)
    mag = torch.einsum("qoi,bqo->biq", R64.abs(), d64.abs())
    assert ((dx.double() - ref).abs() <= 2.0**-8 * ref.abs() + (C + 1) * 2.0**-23 * mag).all()
    ref = torch.einsum("bqo,bqi->qoi", d64, x64)
    mag = torch.einsum("bqo,bqi->qoi", d64.abs(), x64.abs())
    assert ((dR.double() - ref).abs() <= (B + 1) * 2.0**-23 * mag).all()
