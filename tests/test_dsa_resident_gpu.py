"""The diffusion CG with its vectors on chip: one to six vertices a thread (a block owns
a run of 1024 times that), and the general kernel beyond, against the oracle's FP64 CG."""
import numpy as np
import pytest

from helpers import rel_err
from oracle import dsa_oracle as do

pytestmark = pytest.mark.gpu
TOL_CG = 1e-4  # FP32 vectors against the FP64 restatement, relative L2 of the correction


# at 152 blocks: 3-D one, two and three (general kernel) vertices a thread; 2-D two, three, five and seven (general)
@pytest.mark.parametrize("dim,n", [(3, 1), (3, 10), (3, 54), (3, 67), (2, 1), (2, 31), (2, 400), (2, 600), (2, 800),
                                   (2, 980)])
def test_correction_over_vertices_per_thread(dim, n):
    import ouranos_gb300 as og
    if dim == 3:
        p = og.thick_3d(seed=7100 + n, n=n, sn=2, block=1 if n == 1 else n // 2, width=10.0 * n / 64)
    else:
        p = og.heterogeneous_2d(seed=7200 + n, n=n, fe_order=1, sn=2, blocks=1 if n == 1 else 4)
    d = do.Diffusion(p)
    n0 = d.vid.shape[0] * d.nodes
    with og.RadiativeTransfer(p) as rt:
        rt.set_dsa(3)
        v = np.random.default_rng(n).standard_normal(rt.length)
        z = rt.dsa_apply(v)
        ref = d.apply(v, k=3)
        assert rel_err(z[:n0] - v[:n0], ref[:n0] - v[:n0]) < TOL_CG


def test_sums_beyond_the_fp32_range():
    """Every product r z and p q of a step inside the FP32 range, their sums beyond it."""
    import ouranos_gb300 as og
    p = og.thick_3d(seed=7110, n=10, sn=2, block=5, width=100.0 / 64)
    d = do.Diffusion(p)
    n0 = d.vid.shape[0] * d.nodes
    r = np.zeros(d.NV)
    np.add.at(r, d.vid, d.s0[:, None] * d.mix.sum(axis=1)[None, :])  # the right-hand side of v = 1
    z = r / d.diag
    scale = np.sqrt(1e38 / max(np.abs(r * z).max(), np.abs(z * (d.C @ z)).max()))
    assert scale ** 2 * (r @ z) > 1e39 and scale ** 2 * (z @ (d.C @ z)) > 1e39
    with og.RadiativeTransfer(p) as rt:
        rt.set_dsa(1)
        v = np.full(rt.length, scale)
        got = rt.dsa_apply(v)[:n0] - v[:n0]
        assert rel_err(got, d.apply(v, k=1)[:n0] - v[:n0]) < TOL_CG
