"""The default sweep forms (one lane per cell, or several lanes sharing a cell)
against the per-lane and one-warp-per-cell forms of the explicit tilings: every
form rounds every dof in the same order, so the results agree bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(og, dim, order, n, sn, l_max, n_mat=3, groups=1, seed=0, reflect=False):
    rng = np.random.default_rng(1000 * dim + 10 * order + seed)
    q = og.build_quadrature("LS", sn, l_max, dim=dim)
    nc = int(np.prod(n))
    st = rng.uniform(0.5, 20.0, (n_mat, groups))
    ss = rng.uniform(0.0, 0.4, (n_mat, groups, groups, l_max + 1))
    bc = (1, 0, 2, 1, 0, 0)
    return og.Problem(dim, order, n, (0.0,) * dim, tuple(1.0 + 0.5 * a for a in range(dim)), q, st, ss,
                      rng.integers(0, n_mat, nc).astype(np.int32), rng.integers(0, 2, nc).astype(np.int32),
                      np.vstack([np.zeros(groups), rng.uniform(0.5, 1.5, groups)]), bc,
                      rng.uniform(0.2, 2.0, (2 * dim, groups)))


# sides around the tiles of 32, 8, 4 and 2 cells, single planes and single columns
CASES = [
    (2, 1, (33, 31), 4, 0), (2, 1, (31, 1), 4, 1), (2, 1, (65, 7), 8, 3), (2, 1, (1, 9), 4, 0),
    (2, 2, (37, 19), 6, 0), (2, 2, (7, 2), 4, 1), (2, 2, (34, 6), 16, 1),  # the last: one lane per cell
    (2, 3, (9, 11), 4, 1), (2, 3, (5, 3), 4, 3), (2, 4, (9, 5), 4, 1), (2, 5, (5, 4), 4, 0), (2, 5, (2, 3), 4, 1),
    (3, 1, (5, 9, 7), 4, 0), (3, 1, (4, 8, 1), 4, 1), (3, 1, (9, 3, 5), 6, 3),
    (3, 2, (5, 3, 4), 4, 0), (3, 2, (14, 15, 3), 8, 0), (3, 3, (3, 2, 3), 4, 0), (3, 4, (2, 2, 3), 4, 1),
    (3, 5, (2, 1, 2), 2, 0),
]


@pytest.mark.parametrize("dim,order,n,sn,l_max", CASES)
@pytest.mark.parametrize("arith", ["df64_sweep", "df64", "native", "fp32"])
def test_default_form_gives_the_bits_of_the_explicit_tiling(dim, order, n, sn, l_max, arith):
    import ouranos_gb300 as og
    prob = _problem(og, dim, order, n, sn, l_max)
    x = np.random.default_rng(3).standard_normal(prob.vector_length)
    with og.RadiativeTransfer(prob) as rt:
        if arith == "fp32":
            rt.set_precision("fp32")
        else:
            rt.set_fp64_contractions(arith)
        y, b = rt.apply(x), rt.rhs()
        nominal = rt.tiling()
        one_warp = (dim, order) in ((2, 3), (2, 4), (3, 2))  # no per-lane kernel
        rt.set_tiling(*((1, 1, 1) if one_warp else nominal))
        y0, b0 = rt.apply(x), rt.rhs()
        rt.set_tiling()
        assert rt.tiling() == nominal
        y1 = rt.apply(x)
    assert np.isfinite(y).all()
    assert np.array_equal(y, y0)
    assert np.array_equal(b, b0)
    assert np.array_equal(y, y1)


@pytest.mark.parametrize("dim,order,n", [(2, 1, (40, 21)), (2, 2, (24, 23)), (3, 1, (9, 8, 7))])
def test_more_than_256_materials(dim, order, n):
    """The columns' classes no longer fit a byte: they are read plane by plane."""
    import ouranos_gb300 as og
    prob = _problem(og, dim, order, n, 4, 1, n_mat=300)
    x = np.random.default_rng(4).standard_normal(prob.vector_length)
    with og.RadiativeTransfer(prob) as rt:
        for prec in ("fp64", "fp32"):
            rt.set_precision(prec)
            rt.set_tiling()
            y = rt.apply(x)
            rt.set_tiling(*rt.tiling())
            assert np.array_equal(y, rt.apply(x))


@pytest.mark.parametrize("dim,order,n,l_max", [(2, 1, (33, 9), 0), (2, 2, (11, 7), 1), (3, 1, (5, 9, 6), 0)])
def test_time_step_source_and_group_change(dim, order, n, l_max):
    """The expanded source of a time step, and another group's tables."""
    import ouranos_gb300 as og
    prob = _problem(og, dim, order, n, 4, l_max, groups=2)
    gf = np.random.default_rng(5).uniform(0, 1, 2 * prob.vector_length)
    psi = np.random.default_rng(6).uniform(0, 1, prob.quad.n_dir * prob.n_dofs)
    with og.RadiativeTransfer(prob) as rt:
        rt.set_time_step(0.5)
        rt.set_angular_flux(psi)
        rt.set_group(1)
        b = rt.rhs(gf)
        rt.set_tiling(*rt.tiling())
        assert np.array_equal(b, rt.rhs(gf))


@pytest.mark.parametrize("dim,order,n", [(2, 3, (132, 133)), (2, 4, (79, 79)), (3, 2, (13, 13, 14))])
def test_allocation_free_apply_holds_what_the_nominal_tiling_held(dim, order, n):
    """Problems whose scratch only fits with the nominal tiling's edge buffers take
    two lanes per cell, whose tiles are the nominal ones."""
    import ctypes as C

    import torch

    import ouranos_gb300 as og
    from ouranos_gb300 import _capi
    prob = _problem(og, dim, order, n, 4, 0)
    x = torch.from_numpy(np.random.default_rng(8).standard_normal(prob.vector_length)).cuda()
    y = torch.empty_like(x)
    with og.RadiativeTransfer(prob) as rt:
        rc = _capi.lib().ouranos_rt_apply_noalloc(rt._h, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()))
        assert rc == _capi.OK
        ref = rt.apply(x)
        assert torch.equal(y, ref)
        if dim == 2 and order == 3:  # (its fused moment: the one-warp form expands it)
            return
        rt.set_tiling(1, 1, 1)
        assert torch.equal(rt.apply(x), ref)


@pytest.mark.parametrize("dim,order,n", [(2, 1, (70, 9)), (2, 2, (40, 9)), (2, 3, (9, 5)), (3, 1, (9, 17, 5))])
def test_wait_timeout_reports_error_and_recovers(dim, order, n):
    """A dependency wait that cannot be satisfied runs out after the wait limit."""
    import ouranos_gb300 as og
    from ouranos_gb300 import _capi
    prob = _problem(og, dim, order, n, 4, 1)
    x = np.random.default_rng(7).standard_normal(prob.vector_length)
    with og.RadiativeTransfer(prob) as rt:
        ref = rt.apply(x)
        rt.set_wait_limit(2e7)
        rt.debug_wait_bias(1)
        with pytest.raises(_capi.OuranosError) as e:
            rt.apply(x)
        assert e.value.code == _capi.ERR_TIMEOUT
        rt.debug_wait_bias(0)
        rt.set_wait_limit(2e9)
        assert np.array_equal(rt.apply(x), ref)


@pytest.mark.parametrize("dim,order,n,sn", [(2, 2, (34, 6), 16), (3, 1, (5, 9, 7), 4), (3, 3, (3, 2, 3), 4),
                                            (2, 1, (33, 5), 4)])
def test_form_follows_the_arithmetic(dim, order, n, sn):
    """FP64 cell solves take another default form for some orders: switching back and
    forth, with either precision, gives what a fresh handle in that mode gives."""
    import ouranos_gb300 as og
    prob = _problem(og, dim, order, n, sn, 1)
    x = np.random.default_rng(9).standard_normal(prob.vector_length)
    fresh = {}
    for mode in ("df64_sweep", "native", "df64"):
        with og.RadiativeTransfer(prob) as rt:
            rt.set_fp64_contractions(mode)
            rt.set_dsa(2) if order <= 2 else None
            fresh[mode] = rt.apply(x), rt.rhs()
    with og.RadiativeTransfer(prob, precision="fp32") as rt:
        y32 = rt.apply(x)
    with og.RadiativeTransfer(prob) as rt:
        for mode in ("native", "df64_sweep", "df64", "native", "df64_sweep"):
            rt.set_fp64_contractions(mode)
            for _ in range(2):
                assert np.array_equal(rt.apply(x), fresh[mode][0])
            assert np.array_equal(rt.rhs(), fresh[mode][1])
            rt.set_precision("fp32")
            assert np.array_equal(rt.apply(x), y32)
            rt.set_precision("fp64")
