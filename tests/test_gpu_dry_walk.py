"""The dry thermodynamics on grids of more columns than the resident blocks
hold at once (a block then walks over several sets of columns), with ragged
last sets and levels on both sides of the block shapes' changes, against the
FP64 oracle: 1e-12 relative for temperature, alpha and theta in the plain form,
1e-9 in the precision form, and 100 times that for the fields formed by
cancellation or vertical differences (the forms' tolerances elsewhere)."""
import pytest

from helpers import gpu_dv, gpu_sim, gpu_tends, host_case, oracle_sim, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(61, 53, 26), (43, 47, 27), (91, 64, 58), (37, 71, 250)], ids=str)
def test_dry_thermodynamics_over_many_columns(grid):
    nl, rs, f = host_case(case="dry_cbl", nx=grid[0], ny=grid[1], nz=grid[2], dx=50.0, dy=50.0, dz=1500.0 / grid[2])
    o = oracle_sim(nl, rs, f)
    o.update_all_bcs()
    o.th_update()
    for precision, tol in (("fp64", 1e-12), ("fp32", 1e-9)):
        g = gpu_sim(nl, rs, f, precision=precision)
        g.PV.Update_all_bcs(g.Gr)
        g.Th.update(g.Gr, g.RS, g.PV, g.DV)
        d = gpu_dv(g)
        for n in ("temperature", "alpha", "theta"):
            assert rel_l2(d[n], o.dv[n]) < tol, (precision, n)
        for n in ("buoyancy", "buoyancy_frequency"):
            assert rel_l2(d[n], o.dv[n]) < 100 * tol, (precision, n)
        assert rel_l2(gpu_tends(g)["w"], o.tend("w")) < 100 * tol, precision
