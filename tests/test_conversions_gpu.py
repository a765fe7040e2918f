"""The vector kernels' conversions between FP64 and FP32 or pairs: scaling by a power of
two is exact through every one of them, and values at the ends of the FP32 range (zeros,
denormals, values that split into one part only) take the general path."""
import numpy as np
import pytest

from helpers import rel_err

pytestmark = pytest.mark.gpu

# cells per run of 32: less, exactly, one more; every per-cell kernel's size
CASES = [(2, 1, (31, 1), 1), (2, 1, (32, 2), 0), (2, 2, (11, 3), 1), (2, 3, (7, 5), 1), (2, 4, (5, 3), 1),
         (3, 1, (4, 4, 2), 1), (3, 1, (3, 11, 1), 0), (3, 2, (3, 3, 2), 1)]


def _problem(og, dim, order, n, l_max):
    rng = np.random.default_rng(sum(n) + order)
    q = og.build_quadrature("LS", 4, l_max, dim=dim)
    nc = int(np.prod(n))
    st = rng.uniform(0.5, 4.0, (2, 1))
    ss = rng.uniform(0.1, 0.4, (2, 1, 1, l_max + 1))
    return og.Problem(dim, order, n, (0.0,) * dim, (1.0,) * dim, q, st, ss, rng.integers(0, 2, nc).astype(np.int32),
                      np.zeros(nc, np.int32), np.zeros((1, 1)), (0,) * 6, None)


@pytest.mark.parametrize("dim,order,n,l_max", CASES)
def test_scaling_and_range(dim, order, n, l_max):
    import ouranos_gb300 as og
    p = _problem(og, dim, order, n, l_max)
    x = np.random.default_rng(1).standard_normal(p.vector_length)
    ends = x.copy()
    ends[::7] = 0.0
    ends[1::7] = -0.0
    ends[2::7] *= 2.0 ** -75
    ends[3::7] *= 1e-41
    ends[4::7] *= 1e-300
    ends[5::7] = np.float32(1.5)
    with og.RadiativeTransfer(p) as rt:
        rt.set_fp64_contractions("native")
        ref = rt.apply(ends)
        for arith, tol in (("df64_sweep", 1e-12), ("df64", 1e-12), ("fp32", 1e-5)):
            if arith == "fp32":
                rt.set_precision("fp32")
            else:
                rt.set_fp64_contractions(arith)
            y = rt.apply(x)
            for k in (-20, 20):
                assert np.array_equal(rt.apply(x * 2.0 ** k), y * 2.0 ** k)
            assert rel_err(rt.apply(ends), ref) < tol


def test_time_step_source_in_pairs_and_values():
    """The per-direction source of a time step: two rows at a time (even cells) and one,
    in the pair and the FP64 storage."""
    import ouranos_gb300 as og
    for dim, order, n in ((2, 1, (9, 4)), (2, 2, (5, 4)), (3, 1, (5, 3, 4))):
        p = _problem(og, dim, order, n, 0)
        rhs = {}
        psi = np.random.default_rng(6).uniform(0, 1, p.quad.n_dir * p.n_dofs)
        for arith in ("native", "df64", "df64_sweep"):
            with og.RadiativeTransfer(p) as rt:
                rt.set_fp64_contractions(arith)
                rt.set_time_step(2.0)
                rt.set_angular_flux(psi)  # (kept in FP32)
                rhs[arith] = rt.rhs()
        assert np.abs(rhs["native"]).max() > 0
        assert rel_err(rhs["df64"], rhs["native"]) < 1e-12
        assert rel_err(rhs["df64_sweep"], rhs["native"]) < 1e-12
