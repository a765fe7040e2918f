"""A batch whose problems need more sweep kernels than sixteen: every order a batch
takes, every number of fused moments, and both lane counts of the orders that have two
(two lanes where the allocation-free Apply's scratch would not hold the smaller tiles)."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(og, dim, order, n, n_mom):
    rng = np.random.default_rng(100 * dim + 10 * order + n_mom)
    q = og.build_quadrature("LS", 4, 0 if n_mom == 1 else 1, dim=dim)
    if n_mom == 2:
        q = dataclasses.replace(q, m2d=np.ascontiguousarray(q.m2d[:, :2]), d2m=np.ascontiguousarray(q.d2m[:2]),
                                moment_l=np.ascontiguousarray(q.moment_l[:2]))
    nc = int(np.prod(n))
    return og.Problem(dim, order, n, (0.0,) * dim, (1.0,) * dim, q, np.array([[1.0], [4.0]]),
                      rng.uniform(0.0, 0.4, (2, 1, 1, q.l_max + 1)), rng.integers(0, 2, nc).astype(np.int32),
                      rng.integers(0, 2, nc).astype(np.int32), np.array([[0.0], [1.0]]), (1,) + (0,) * (2 * dim - 1),
                      np.ones((2 * dim, 1)))


CLASSES = [(2, 1, (9, 7), 1), (2, 1, (9, 7), 2), (2, 1, (9, 7), 3), (2, 2, (7, 5), 1), (2, 2, (7, 5), 2),
           (2, 2, (7, 5), 3), (2, 3, (5, 6), 1), (2, 3, (132, 133), 1), (2, 3, (5, 6), 3), (2, 3, (92, 92), 3),
           (2, 4, (4, 3), 1), (2, 4, (79, 79), 1), (3, 1, (5, 3, 4), 1), (3, 1, (5, 3, 4), 2), (3, 1, (5, 3, 4), 4),
           (3, 2, (3, 2, 3), 1), (3, 2, (13, 13, 14), 1)]


def test_seventeen_classes():
    import ouranos_gb300 as og
    probs = [_problem(og, *c) for c in CLASSES]
    with og.Batch(probs) as b:
        x = np.random.default_rng(1).standard_normal(b.length)
        y, r, y32 = b.apply(x), b.rhs(), b.apply(x, precision="fp32")
        assert np.array_equal(b.apply(x), y)  # (the captured graph)
        for p, xs, ys, rs, fs in zip(probs, b.slices(x), b.slices(y), b.slices(r), b.slices(y32)):
            with og.RadiativeTransfer(p) as rt:
                rt.set_fp64_contractions("df64")
                assert np.array_equal(rt.apply(np.ascontiguousarray(xs)), ys)
                assert np.array_equal(rt.rhs(), rs)
                rt.set_precision("fp32")
                assert np.array_equal(rt.apply(np.ascontiguousarray(xs)), fs)
