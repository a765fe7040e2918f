"""The columns' sigma_t classes, packed four planes to a word on the device, against the
kernels that read them cell by cell: another map of materials to classes in each group,
plane counts around a word, single columns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(2, (33, 1)), (2, (5, 3)), (2, (1, 4)), (2, (40, 5)), (2, (3, 8)), (2, (2, 9)),
                                   (3, (5, 9, 1)), (3, (4, 3, 4)), (3, (1, 1, 7)), (3, (3, 2, 13))])
def test_classes_of_every_group(dim, n):
    import ouranos_gb300 as og
    rng = np.random.default_rng(sum(n))
    q = og.build_quadrature("LS", 4, 1, dim=dim)
    nc = int(np.prod(n))
    st = np.array([[1.0, 2.0, 5.0], [2.0, 2.0, 3.0], [4.0, 1.0, 5.0], [1.0, 3.0, 3.0]])
    p = og.Problem(dim, 1, n, (0.0,) * dim, (1.0,) * dim, q, st, rng.uniform(0.0, 0.2, (4, 3, 3, 2)),
                   rng.integers(0, 4, nc).astype(np.int32), np.zeros(nc, np.int32), np.ones((1, 3)), (0,) * (2 * dim),
                   np.zeros((2 * dim, 3)))
    x = rng.standard_normal(p.vector_length)
    out = []
    with og.RadiativeTransfer(p) as rt:
        for hook in (0, 1):
            rt.debug_nominal_form(hook)
            assert rt.form()[4] == (hook == 0)
            for g in (0, 1, 2, 1, 0):
                rt.set_group(g)
                out.append(rt.apply(x))
    for a, b in zip(out[:5], out[5:]):
        assert np.array_equal(a, b)
    assert np.array_equal(out[0], out[4]) and not np.array_equal(out[0], out[1])
