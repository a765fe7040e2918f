"""Right-hand sides with another inflow on every face, by the sweep's default forms, at
the sides where a warp's tile begins and ends: the first cells of a tile take the
boundary's value, the next tile's first cells the neighbour's."""
import numpy as np
import pytest

from helpers import rel_err
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

# FP64: the parity bar of the other tests; FP32: a right-hand side is a sum of some
# (cells along an axis) x (dofs of a cell) rounded terms, 100 x 125 x 6e-8
TOL = {"df64_sweep": 1e-12, "native": 1e-12, "fp32": 1e-5}

# one lane per cell (2-D tiles of 32 x 1, 3-D 4 x 8), then several lanes per cell
CASES = [(2, 1, (31, 1), 4), (2, 1, (32, 2), 4), (2, 1, (33, 31), 4), (2, 2, (34, 6), 16), (2, 2, (65, 3), 16),
         (3, 1, (4, 8, 1), 4), (3, 1, (5, 9, 7), 4), (3, 1, (9, 17, 3), 4),
         (2, 2, (9, 5), 4), (2, 3, (9, 5), 4), (2, 5, (3, 4), 4), (3, 2, (5, 3, 4), 4), (3, 3, (3, 2, 3), 4)]


@pytest.mark.parametrize("dim,order,n,sn", CASES)
@pytest.mark.parametrize("arith", sorted(TOL))
def test_rhs_with_inflow_matches_oracle(dim, order, n, sn, arith):
    import ouranos_gb300 as og
    rng = np.random.default_rng(100 * dim + order)
    q = og.build_quadrature("LS", sn, 1, dim=dim)
    nc = int(np.prod(n))
    prob = og.Problem(dim, order, n, (0.0,) * dim, tuple(1.0 + 0.3 * a for a in range(dim)), q,
                      rng.uniform(0.5, 4.0, (3, 1)), rng.uniform(0.0, 0.3, (3, 1, 1, 2)),
                      rng.integers(0, 3, nc).astype(np.int32), rng.integers(0, 2, nc).astype(np.int32),
                      np.array([[0.0], [0.7]]), (1, 1, 2, 1, 1, 2), 0.5 + np.arange(2 * dim)[:, None])
    ref = po.OracleProblem(prob.arrays()).rhs()
    with og.RadiativeTransfer(prob) as rt:
        if arith == "fp32":
            rt.set_precision("fp32")
        else:
            rt.set_fp64_contractions(arith)
        b = rt.rhs()
        again = [rt.rhs() for _ in range(3)]
    assert rel_err(b, ref) < TOL[arith]
    for c in again:
        assert np.array_equal(b, c)
