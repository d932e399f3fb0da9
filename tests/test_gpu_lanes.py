"""The advection kernels on level counts around the warp's 31 and 32 cells and
the diffusion kernels on counts around their 128-level rows, on both sides of
the rules that map threads to rows or to the flattened plane, and with marching
chunks of one cell up, against the FP64 oracle: advection tendencies 1e-10 (the
plain form's), 1e-5 (FP32 weights); diffusion 1e-12."""
import ctypes

import numpy as np
import pytest

from helpers import gpu_dv, gpu_sim, gpu_tends, host_case, oracle_sim, rel_l2
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


# 128-level rows leave no thread idle (128), few (124, 127, 252: by rows) or more (flat)
LEVELS = [(7, 6, 33), (5, 9, 122), (6, 4, 124), (4, 7, 127), (9, 5, 128), (4, 5, 252), (5, 4, 240)]


@pytest.mark.parametrize("case", ["bomex", "bomex_no_source", "dry_cbl"])
@pytest.mark.parametrize("grid", LEVELS, ids=lambda g: "x".join(map(str, g)))
def test_diffusion_lane_maps(grid, case):
    from oracle.sgs import OracleSGS, scheme_from_namelist
    nl, rs, f = host_case(case=case.split("_no")[0], nx=grid[0], ny=grid[1], nz=grid[2], dx=100.0, dy=100.0, dz=20.0)
    f = _stir(f)
    nl = dict(nl, sgs={"scheme": "Smagorinsky"}, diffusion={"qt_entropy_source": case == "bomex"})
    g, o = gpu_sim(nl, rs, f), oracle_sim(nl, rs, f)
    o.update_all_bcs()
    g.PV.Update_all_bcs(g.Gr)
    o.th_update()
    g.Th.update(g.Gr, g.RS, g.PV, g.DV)
    sgs = OracleSGS(scheme_from_namelist(nl), o.d, np.zeros(g.Gr.shape[2]))
    sgs.ke_update(o)
    sgs.sgs_update(o)
    g.SGS.update(g.Gr, g.DV, g.PV, g.Ke)
    sh, d = g.Gr.shape, gpu_dv(g)
    for n, a, b in (("strain", g.Ke.strain_rate_mag.cpu().numpy(), sgs.strain_rate_mag),
                    ("viscosity", d["viscosity"], sgs.viscosity), ("diffusivity", d["diffusivity"], sgs.diffusivity)):
        assert rel_l2(a.reshape(sh)[2:], b.reshape(sh)[2:]) < 1e-12, n
    for update, oracle_update in ((lambda: g.SD.update(g.Gr, g.RS, g.PV, g.DV), sgs.sd_update),
                                  (lambda: g.MD.update(g.Gr, g.RS, g.PV, g.DV, g.Ke), sgs.md_update)):
        o.tendencies[:] = 0.0
        g.PV.tendencies.zero_()
        oracle_update(o)
        update()
        t = gpu_tends(g)
        for n in o.names:
            assert rel_l2(t[n], o.tend(n)) < 1e-12, (oracle_update.__name__, n)


@pytest.mark.parametrize("nz", [122, 127, 33])
def test_scalar_diffusion_of_three_scalars(nz):
    """s, qt with its entropy source and a third scalar take the general
    kernel: the tendencies of s and qt as the pair's, the third's (equal to
    qt) as qt's."""
    import torch
    from pycles_b200 import _capi
    nl, rs, f = host_case(case="bomex", nx=6, ny=5, nz=nz, dx=100.0, dy=100.0, dz=20.0)
    nl = dict(nl, sgs={"scheme": "Smagorinsky"}, diffusion={"qt_entropy_source": True})
    g = gpu_sim(nl, rs, _stir(f))
    Gr, PV, DV, RS = g.Gr, g.PV, g.DV, g.RS
    PV.Update_all_bcs(Gr)
    g.Th.update(Gr, RS, PV, DV)
    g.SGS.update(Gr, DV, PV, g.Ke)
    PV.tendencies.zero_()
    g.SD.update(Gr, RS, PV, DV)
    want = gpu_tends(g)
    x = [PV.field("s", Gr), PV.field("qt", Gr), PV.field("qt", Gr).clone()]
    t = [torch.zeros_like(v) for v in x]
    p3 = ctypes.c_void_p * 3
    rc = _capi.load().pb_scalar_diffusion(
        ctypes.byref(Gr.dims), _capi.ptr(RS.d_rho0), _capi.ptr(RS.d_rho0_half), _capi.ptr(RS.d_alpha0_half),
        _capi.ptr(DV.field("diffusivity", Gr)), 3, p3(*map(_capi.ptr, x)), p3(*map(_capi.ptr, t)), None, 1, 0,
        _capi.ptr(RS.d_p0_half), _capi.ptr(DV.field("qv", Gr)), _capi.ptr(DV.field("temperature", Gr)),
        _capi.stream_handle())
    _capi.check(rc, "pb_scalar_diffusion")
    for name, got in zip(("s", "qt", "qt"), t):
        np.testing.assert_array_equal(got.cpu().numpy(), want[name])
