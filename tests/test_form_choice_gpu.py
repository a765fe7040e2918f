"""Which kernel a handle's sweeps run in: a tiling that is read and set again keeps it,
and the kernels of the nominal tilings, reached through the test hook, give the
default forms' bits and the oracle's values."""
import numpy as np
import pytest

from helpers import rel_err
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _problem(og, dim, order, n, sn=4, l_max=1):
    rng = np.random.default_rng(1000 * dim + 10 * order)
    q = og.build_quadrature("LS", sn, l_max, dim=dim)
    nc = int(np.prod(n))
    return og.Problem(dim, order, n, (0.0,) * dim, tuple(1.0 + 0.5 * a for a in range(dim)), q,
                      rng.uniform(0.5, 6.0, (3, 1)), rng.uniform(0.0, 0.4, (3, 1, 1, l_max + 1)),
                      rng.integers(0, 3, nc).astype(np.int32), rng.integers(0, 2, nc).astype(np.int32),
                      np.array([[0.0], [1.0]]), (1, 0, 2, 1, 0, 0), rng.uniform(0.2, 2.0, (2 * dim, 1)))


def _set(rt, arith):
    if arith == "fp32":
        rt.set_precision("fp32")
    else:
        rt.set_fp64_contractions(arith)


# (problem, the default form's lanes per cell)
FORMS = [((2, 1, (33, 9)), 1), ((2, 2, (9, 5)), 4), ((2, 2, (66, 6), 16), 1), ((2, 3, (9, 5)), 8), ((2, 4, (5, 4)), 8),
         ((2, 5, (4, 3)), 16), ((3, 1, (5, 9, 7)), 1), ((3, 2, (5, 3, 4)), 16), ((3, 3, (3, 2, 3)), 16),
         ((3, 4, (2, 2, 3)), 32), ((3, 5, (2, 1, 2), 2), 32)]


@pytest.mark.parametrize("prob,lanes", FORMS)
def test_a_tiling_read_and_set_again_keeps_the_form(prob, lanes):
    import ouranos_gb300 as og
    with og.RadiativeTransfer(_problem(og, *prob)) as rt:
        for mode in ("df64_sweep", "native"):
            rt.set_fp64_contractions(mode)
            form, tiling = rt.form(), rt.tiling()
            if mode == "df64_sweep":
                assert form[3:] == (lanes, True)
            rt.set_tiling(*tiling)
            assert rt.form() == form and rt.tiling() == tiling
            rt.set_tiling(1, 1, 1)
            rt.set_tiling(*tiling)
            assert rt.form() == form and rt.tiling() == tiling


@pytest.mark.parametrize("prob", [f[0] for f in FORMS if f[0][:2] not in ((2, 3), (2, 4), (3, 2))])
@pytest.mark.parametrize("arith", ["df64_sweep", "df64", "fp32"])
def test_nominal_kernels_give_the_default_forms_bits(prob, arith):
    import ouranos_gb300 as og
    p = _problem(og, *prob)
    x = np.random.default_rng(3).standard_normal(p.vector_length)
    with og.RadiativeTransfer(p) as rt:
        _set(rt, arith)
        y, b = rt.apply(x), rt.rhs()
        before = rt.form()
        rt.debug_nominal_form(1)
        cx, cy, dirs, lanes, default = rt.form()
        assert (cx, cy, dirs) == rt.tiling() and not default
        assert np.array_equal(rt.apply(x), y) and np.array_equal(rt.rhs(), b)
        rt.debug_nominal_form(0)
        assert rt.form() == before
        assert np.array_equal(rt.apply(x), y)


@pytest.mark.parametrize("prob", [f[0] for f in FORMS if (f[0][0] == 2 and f[0][1] == 5) or (f[0][0] == 3 and f[0][1] >= 3)])
def test_one_warp_per_cell_matches_oracle_and_reports_its_timeouts(prob):
    """The orders whose nominal tiling is one warp per cell, in that form."""
    import ouranos_gb300 as og
    from ouranos_gb300 import _capi
    p = _problem(og, *prob)
    x = np.random.default_rng(5).standard_normal(p.vector_length)
    O = po.OracleProblem(p.arrays())
    ref, rhs = O.apply(x), po.OracleProblem(p.arrays()).rhs()
    with og.RadiativeTransfer(p) as rt:
        rt.debug_nominal_form(1)
        assert rt.form() == (1, 1, 1, 32, False)
        assert rel_err(rt.apply(x), ref) < 1e-12 and rel_err(rt.rhs(), rhs) < 1e-12
        rt.set_wait_limit(2e7)
        rt.debug_wait_bias(1)
        with pytest.raises(_capi.OuranosError) as e:
            rt.apply(x)
        assert e.value.code == _capi.ERR_TIMEOUT
        rt.debug_wait_bias(0)
        rt.set_wait_limit(2e9)
        assert rel_err(rt.apply(x), ref) < 1e-12
        rt.set_precision("fp32")
        assert rel_err(rt.apply(x), ref) < 1e-5 and rel_err(rt.rhs(), rhs) < 1e-5


def test_autotuned_tilings_of_orders_that_choose_their_lanes():
    """Their tilings all run the same kernel: nothing is timed, the nominal one comes back."""
    import ouranos_gb300 as og
    probs = [_problem(og, 2, 3, (9, 5)), _problem(og, 2, 4, (5, 4)), _problem(og, 3, 2, (5, 3, 4))]
    with og.Batch(probs) as b:
        assert b.autotune(reps=1).tolist() == [[16, 1, 1], [16, 1, 1], [4, 4, 1]]


# (problem, directions' |Omega| classes): a task queue per class, below and above a warp's 32
@pytest.mark.parametrize("dim,order,n,sn,mats", [(2, 3, (17, 5), 16, 64), (2, 4, (9, 4), 16, 16), (2, 5, (5, 4), 16, 8),
                                                 (3, 2, (5, 4, 3), 8, 16), (3, 3, (3, 2, 2), 4, 4)])
def test_task_queues_give_one_warp_per_cells_bits(dim, order, n, sn, mats):
    import ouranos_gb300 as og
    rng = np.random.default_rng(dim + order)
    q = og.build_quadrature("LS", sn, 1, dim=dim)
    nc = int(np.prod(n))
    p = og.Problem(dim, order, n, (0.0,) * dim, (1.0,) * dim, q, rng.uniform(0.5, 5.0, (mats, 1)),
                   rng.uniform(0.0, 0.2, (mats, 1, 1, 2)), rng.integers(0, mats, nc).astype(np.int32),
                   np.zeros(nc, np.int32), np.ones((1, 1)), (1,) * (2 * dim), np.ones((2 * dim, 1)))
    x = rng.standard_normal(p.vector_length)
    with og.RadiativeTransfer(p) as rt:
        for precision in ("fp64", "fp32"):
            rt.set_precision(precision)
            rt.set_tiling()
            assert rt.form()[4] and rt.form()[3] > 1
            y, b = [rt.apply(x) for _ in range(3)], rt.rhs()
            if (dim, order) in ((2, 3), (2, 4), (3, 2)):
                rt.set_tiling(1, 1, 1)
            else:
                rt.debug_nominal_form(1)
            assert rt.form()[3:] == (32, False)
            ref = rt.apply(x)
            assert all(np.array_equal(v, ref) for v in y)
            assert np.array_equal(b, rt.rhs())
            rt.debug_nominal_form(0)


def test_many_materials_side_by_side_share_cells():
    """2-D Q2: four lanes to a cell where a row of 32 cells meets many materials, in any
    order, one lane where they come in blocks; the same bits."""
    import ouranos_gb300 as og
    rng = np.random.default_rng(8)
    q = og.build_quadrature("LS", 16, 1, dim=2)
    n = (66, 5)
    cells = np.arange(n[0] * n[1])
    x = None
    for mat, lanes in ((cells % 16, 4), (rng.integers(0, 16, cells.size), 4), (cells % 66 // 6, 1), (cells % 2, 1)):
        p = og.Problem(2, 2, n, (0.0, 0.0), (1.0, 1.0), q, rng.uniform(0.5, 5.0, (16, 1)),
                       rng.uniform(0.0, 0.2, (16, 1, 1, 2)), mat.astype(np.int32), np.zeros(cells.size, np.int32),
                       np.ones((1, 1)), (1,) * 4, np.ones((4, 1)))
        x = rng.standard_normal(p.vector_length)
        with og.RadiativeTransfer(p) as rt:
            assert rt.form()[3:] == (lanes, True)
            y, b = rt.apply(x), rt.rhs()
            rt.debug_nominal_form(1)
            assert np.array_equal(rt.apply(x), y) and np.array_equal(rt.rhs(), b)
