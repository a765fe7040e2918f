"""Device results written straight into the caller's vector, or through the library's own
where that is not possible: the same vector, overlapping ones, odd addresses."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("order", [False, True])
def test_targets(precision, order):
    import torch

    import ouranos_gb300 as og
    p = og.heterogeneous_2d(seed=5, n=12, fe_order=1, sn=4, l_max=1, g_aniso=0.3, blocks=3)
    if order:
        import dataclasses
        p = dataclasses.replace(p, cell_order=np.random.default_rng(3).permutation(144))
    n = p.vector_length
    x = np.random.default_rng(2).standard_normal(n)
    with og.RadiativeTransfer(p, precision=precision) as rt:
        rt.set_dsa(3)
        ref, rhs, z = rt.apply(x), rt.rhs(out=x.copy()), rt.dsa_apply(x)
        buf = torch.zeros(2 * n + 8, dtype=torch.float64, device="cuda")
        for at_x, at_y in ((0, n), (0, 0), (3, n + 4), (0, 1), (5, 0), (0, n + 1), (n, 0)):
            for call, want in ((lambda u, v: rt.Apply(u, v), ref), (lambda u, v: rt.dsa_apply(u, out=v), z)):
                buf.zero_()
                xv, yv = buf[at_x:at_x + n], buf[at_y:at_y + n]
                xv.copy_(torch.from_numpy(x))
                call(xv, yv)
                assert np.array_equal(yv.cpu().numpy(), want)
        v = torch.from_numpy(x).cuda()
        assert np.array_equal(rt.rhs(out=v).cpu().numpy(), rhs)
