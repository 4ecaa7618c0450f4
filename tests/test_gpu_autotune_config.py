"""The grouped autotuner returns a configuration of its documented values in every
field, schedule and store included."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("rep", range(4))
def test_grouped_autotune_sets_every_field(rep):
    from jaxfun_gb300 import _lib
    from jaxfun_gb300.la.helmholtz import UnevenHelmholtzSolver

    S = UnevenHelmholtzSolver("chebyshev", np.array([18, 34, 34, 66, 130]), np.ones(5))
    S.autotune(reps=1)
    assert S.cfg.operand_a_in_tmem in (0, 1) and S.cfg.order in (0, 1, 2)
    assert S.cfg.ctas == 0 and S.cfg.stages in (0, 2, 3) and S.cfg.mtile in (0, 64)
    assert S.cfg.schedule == 0 and S.cfg.store == 0
    assert C.sizeof(_lib.TcConfig) == 7 * C.sizeof(C.c_int)
