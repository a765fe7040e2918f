"""The allocation-free Apply's limit counts two tagged words to an edge value in FP32 too."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 2-D Q1, LS S4, P0, tiles of 8 x 1 x 4 in FP32: 272 bytes a cell at two words, 248 at one, of 32 MiB
@pytest.mark.parametrize("side,fits", [(344, True), (360, False)])
def test_limit_of_an_explicit_tiling(side, fits):
    import torch

    import ouranos_gb300 as og
    from ouranos_gb300 import _capi
    q = og.build_quadrature("LS", 4, 0, dim=2)
    p = og.uniform_problem(2, 1, (side, side), (0.0, 0.0), (1.0, 1.0), q, 1.0, 0.5, 1.0)
    x = torch.from_numpy(np.random.default_rng(2).standard_normal(p.vector_length)).cuda()
    y = torch.empty_like(x)
    with og.RadiativeTransfer(p, precision="fp32") as rt:
        rt.set_tiling(8, 1, 4)
        rc = _capi.lib().ouranos_rt_apply_noalloc(rt._h, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()))
        if not fits:
            assert rc == _capi.ERR_BAD_INPUT and "scratch" in _capi.last_error(rt._h)
            return
        assert rc == _capi.OK
        assert torch.equal(y, rt.apply(x))
