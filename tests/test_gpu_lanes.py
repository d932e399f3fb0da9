"""The advection and diffusion kernels on level counts around the warp's 31
and 32 cells, on both sides of the rule that maps threads to rows or to the
flattened plane, and with marching chunks of one cell up, against the FP64
oracle: tendencies 1e-10 (the plain form's), 1e-5 (FP32 weights)."""
import pytest

from helpers import gpu_sim, gpu_tends, host_case, oracle_sim, rel_l2
from test_gpu_precision import _stir

pytestmark = pytest.mark.gpu

GRIDS = [(5, 4, 30), (7, 6, 31), (6, 9, 32), (4, 5, 33), (9, 8, 40), (33, 5, 62), (6, 7, 64), (8, 37, 75)]


@pytest.mark.parametrize("order,gw", [(5, 3), (7, 4)])
@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g)))
def test_advection_lane_maps(grid, order, gw):
    nl, rs, f = host_case(case="bomex", nx=grid[0], ny=grid[1], nz=grid[2], dx=100.0, dy=100.0, dz=40.0, gw=gw,
                          scalar_order=order)
    f = _stir(f)
    o = oracle_sim(nl, rs, f)
    o.update_all_bcs()
    o.sa_update()
    o.ma_update()
    for precision, tol in (("fp64", 1e-10), ("fp32", 1e-5)):
        g = gpu_sim(nl, rs, f, precision=precision)
        g.PV.Update_all_bcs(g.Gr)
        g.SA.update(g.Gr, g.RS, g.PV, g.DV)
        g.MA.update(g.Gr, g.RS, g.PV)
        t = gpu_tends(g)
        for n in o.names:
            assert rel_l2(t[n], o.tend(n)) < tol, (precision, n)
