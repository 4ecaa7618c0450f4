"""Tensor-core contraction, stores from registers: clipped tiles (operator rows,
input rows, contracted extent) against FP64, with nothing written outside."""

import numpy as np
import pytest
import torch

from jaxfun_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["tf32", "bf16x3"])
@pytest.mark.parametrize("B,M,P,K", [(3, 17, 33, 32), (2, 129, 130, 64), (5, 100, 127, 96),
                                     (1, 250, 260, 256), (40, 36, 129, 128)])
def test_clipped_tiles(prec, B, M, P, K):
    """Split TF32 keeps 2^-21 of a product, split BF16 2^-15, and the FP32 sums add
    K 2^-23 of the terms."""
    from jaxfun_gb300.la import split_tf32
    from jaxfun_gb300.la.mixed import split_bf16

    L = _lib.lib()
    op = np.random.default_rng(M).standard_normal((M, K))
    g = torch.Generator(device="cuda")
    g.manual_seed(P)
    x = torch.randn(B, P, K, device="cuda", generator=g)
    ld = P + 8
    out = torch.full((B, M + 2, ld), 7.0, device="cuda")
    hi, lo = split_tf32(op) if prec == "tf32" else split_bf16(op)
    d = _lib.ContractDesc(batch=B, nseg=1, M=M, P=P, K=K, op_ld=K, in_ld=K, in_batch=P * K,
                          out_ld=ld, out_batch=(M + 2) * ld, alpha=1.0, beta=0.0)
    call = L.jfg_contract_tc if prec == "tf32" else L.jfg_contract_tc_bf16x3
    st = call(d, hi.data_ptr(), lo.data_ptr(), x.data_ptr(), out[:, 1].data_ptr(),
              _lib.stream_handle())
    assert st == 0, _lib.status_string(st)
    torch.cuda.synchronize()
    assert L.jfg_device_status() == 0
    A = torch.as_tensor(op, device="cuda")
    ref, mag = A @ x.double().mT, A.abs() @ x.double().abs().mT
    eps = 2.0 ** (-21 if prec == "tf32" else -15) + K * 2.0**-23
    assert ((out[:, 1:-1, :P].double() - ref).abs() <= eps * mag).all()
    assert (out[:, 0] == 7.0).all() and (out[:, -1] == 7.0).all() and (out[..., P:] == 7.0).all()
