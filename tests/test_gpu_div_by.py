"""Division by a divisor whose reciprocal is kept (csrc/pb_common.cuh), over the
divisors that the kernels use and around powers of two, for quotients of every
magnitude, near half-way cases, zeros, infinities and NaNs: div_by_normal has
the bits of `/` on the range that it states and wherever quotient_normal takes
its result; and its callers on unusual inputs: the pressure solve's divergence,
the dry thermodynamics and the entropy source of the total-water diffusion.
Tolerance: none (equality; NaNs are equal) but for the last, 1e-12."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from helpers import ROOT, gpu_dv, gpu_sim, gpu_tends, host_case, oracle_sim, rel_l2

pytestmark = pytest.mark.gpu

PROBE = r"""
#include "pb_common.cuh"
__global__ void probe(const double* a, const double* b, double* q, double* r, double* d, long long n) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  r[i] = div_by_normal(a[i], b[i], 1.0 / b[i]);
  q[i] = quotient_normal(r[i]) ? r[i] : a[i] / b[i];
  d[i] = a[i] / b[i];
}
extern "C" int run_probe(const double* a, const double* b, double* q, double* r, double* d, long long n) {
  probe<<<(unsigned)((n + 255) / 256), 256>>>(a, b, q, r, d, n);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def probe_lib(tmp_path_factory):
    d = str(tmp_path_factory.mktemp("div_by"))
    src, so = os.path.join(d, "probe.cu"), os.path.join(d, "probe.so")
    with open(src, "w") as f:
        f.write(PROBE)
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared",
                    "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "pycles_b200", "csrc"), src, "-o", so],
                   check=True)
    return ctypes.CDLL(so)


def _operands():
    rng = np.random.default_rng(17)
    two = 2.0 ** np.arange(-40, 41, dtype=np.float64)
    b = np.concatenate([
        [100000.0, 298.15, 1004.0, 3.0, 7.0, 1.0],                             # p_tilde, T_tilde, cpd
        rng.uniform(0.75, 3.0, 40), rng.uniform(2.0e4, 1.1e5, 40), rng.uniform(0.6, 1.1, 40),  # alpha0, p0, Exner
        two, np.nextafter(two, 0.0), np.nextafter(two, np.inf), -rng.uniform(0.5, 2.0, 10),
        [0.0, -0.0, np.inf, -np.inf, np.nan],
    ])
    q = np.concatenate([
        rng.uniform(-4.0, 4.0, 400), np.ldexp(rng.uniform(1.0, 2.0, 1200), rng.integers(-1074, 1024, 1200)),
        np.ldexp(1.0, rng.integers(-1074, 1024, 200)), -np.ldexp(rng.uniform(1.0, 2.0, 200), rng.integers(-40, 40, 200)),
    ])
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2250738585072014e-308,
                        1.7976931348623157e308, -1.7976931348623157e308])
    with np.errstate(all="ignore"):
        A = [np.broadcast_to(q, (b.size, q.size)).ravel(), (q * b[:, None]).ravel()]
        # dividends next to a quotient's half-way points
        h = np.ldexp(rng.integers(2 ** 52, 2 ** 53, 400).astype(np.float64), -52)
        A.append(((h + np.spacing(h) / 2) * b[:, None]).ravel())
        A.append((np.nextafter(h, 4.0) * b[:, None]).ravel())
        A.append(np.broadcast_to(special, (b.size, special.size)).ravel())
    B = [np.broadcast_to(b[:, None], (b.size, a.size // b.size)).ravel() for a in A]
    return np.concatenate(A), np.concatenate(B)


def test_div_by_is_division(probe_lib):
    import torch
    a, b = _operands()
    at, bt = torch.as_tensor(a, device="cuda"), torch.as_tensor(b, device="cuda")
    q, r, d = (torch.empty_like(at) for _ in range(3))
    assert probe_lib.run_probe(*[ctypes.c_void_p(t.data_ptr()) for t in (at, bt, q, r, d)],
                               ctypes.c_longlong(a.size)) == 0
    q, r, d = (t.cpu().numpy() for t in (q, r, d))
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(d, a / b)
    differ = lambda x: (x.view(np.int64) != d.view(np.int64)) & ~(np.isnan(x) & np.isnan(d))  # noqa: E731
    show = lambda bad: [(a[i], b[i], q[i], r[i], d[i]) for i in np.nonzero(bad)[0][:5]]  # noqa: E731
    assert not differ(q).any(), show(differ(q))
    divisor = (np.abs(b) >= 2.0 ** -60) & (np.abs(b) <= 2.0 ** 1000)
    bad = differ(r) & divisor & (np.abs(d) >= 2.0 ** -900) & (np.abs(d) <= 2.0 ** 1022)
    assert not bad.any(), show(bad)
    assert np.all(r[divisor & (a == 0.0)] == 0.0) and np.all(np.isnan(r[divisor & ~np.isfinite(a)]))


def test_divergence_of_unusual_velocities():
    import torch
    nl, rs, _ = host_case(case="dry_cbl", nx=8, ny=6, nz=10, dx=50.0, dy=50.0, dz=50.0)
    sim = gpu_sim(nl, rs, {})
    Gr, PV = sim.Gr, sim.PV
    rng = np.random.default_rng(2)
    u, v = rng.standard_normal(Gr.shape), rng.standard_normal(Gr.shape)
    u[5, 4, 6], u[7, 5, 8] = np.inf, -np.inf
    v[4, 5, 9] = np.inf
    u[:, 7] *= 1e-306
    v[:, 7:9] *= 1e-306
    for n, x in (("u", u), ("v", v)):
        PV.get_variable_array(n, Gr).copy_(torch.as_tensor(x))
    PV.get_variable_array("w", Gr).zero_()
    sim.Pr.solve(Gr, sim.RS, sim.DV, PV)
    g, inner = Gr.dims.gw, (slice(Gr.dims.gw, -Gr.dims.gw),) * 3
    ah = rs["alpha0_half"]
    with np.errstate(all="ignore"):
        want = np.zeros(Gr.shape)
        want[1:] += (u[1:] / ah - u[:-1] / ah) * Gr.dims.dxi[0]
        want[:, 1:] += (v[:, 1:] / ah - v[:, :-1] / ah) * Gr.dims.dxi[1]
    got = sim.DV.get_variable_array("divergence", Gr).cpu().numpy()
    assert np.isinf(want[inner]).sum() == 6
    np.testing.assert_array_equal(got[inner], want[inner])


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_dry_thermodynamics_of_infinite_entropy(precision):
    nl, rs, f = host_case(case="dry_cbl", nx=6, ny=5, nz=9, dx=50.0, dy=50.0, dz=50.0)
    sim = gpu_sim(nl, rs, f, precision=precision)
    s = sim.PV.get_variable_array("s", sim.Gr)
    s[4, 4, 5], s[5, 4, 7], s[6, 6, 6] = -np.inf, np.inf, np.nan
    sim.Th.update(sim.Gr, sim.RS, sim.PV, sim.DV)
    d = {n: x.reshape(sim.Gr.shape) for n, x in gpu_dv(sim).items()}
    for n in ("temperature", "alpha", "theta"):
        assert d[n][4, 4, 5] == 0.0 and d[n][5, 4, 7] == np.inf and np.isnan(d[n][6, 6, 6]), n


def test_entropy_source_of_dry_and_tiny_vapour(monkeypatch):
    """Cells without vapour (qv = 0, log of zero) and with qv = 1e-300 beside
    ordinary ones: the entropy tendency of ScalarDiffusion against the oracle."""
    import math

    import torch
    from oracle import port
    from oracle.sgs import OracleSGS, scheme_from_namelist
    log = lambda x: math.log(x) if x > 0.0 else (-math.inf if x == 0.0 else math.nan)  # noqa: E731  (as C's)
    monkeypatch.setattr(port, "_vlog", np.frompyfunc(log, 1, 1))
    nl, rs, f = host_case(case="bomex", nx=8, ny=7, nz=12)
    nl = dict(nl, sgs={"scheme": "UniformViscosity", "UniformViscosity": {"diffusivity": 5.0, "viscosity": 5.0}},
              diffusion={"qt_entropy_source": True})
    g, o = gpu_sim(nl, rs, f), oracle_sim(nl, rs, f)
    sh = g.Gr.shape
    rng = np.random.default_rng(4)
    o.update_all_bcs()
    g.PV.Update_all_bcs(g.Gr)
    o.th_update()
    g.Th.update(g.Gr, g.RS, g.PV, g.DV)
    qv = o.dv["qv"].reshape(sh) * (1.0 + 0.1 * rng.standard_normal(sh))
    qv[4], qv[6] = 0.0, 1e-300
    o.dv["qv"][:] = qv.ravel()
    g.DV.get_variable_array("qv", g.Gr).copy_(torch.as_tensor(qv))
    qt = o.var("qt").reshape(sh)
    qt *= 1.0 + 0.01 * rng.standard_normal(sh)
    g.PV.get_variable_array("qt", g.Gr).copy_(torch.as_tensor(qt.copy()))
    sgs = OracleSGS(scheme_from_namelist(nl), o.d, np.zeros(sh[2]))
    o.tendencies[:] = 0.0
    g.PV.tendencies.zero_()
    with np.errstate(all="ignore"):
        sgs.ke_update(o)
        sgs.sgs_update(o)
        sgs.sd_update(o)
    g.SGS.update(g.Gr, g.DV, g.PV, g.Ke)
    g.SD.update(g.Gr, g.RS, g.PV, g.DV)
    got, want = gpu_tends(g), {n: o.tend(n) for n in ("s", "qt")}
    for n in ("s", "qt"):
        a, b = got[n].reshape(sh), want[n].reshape(sh)
        for x in (np.isnan, np.isposinf, np.isneginf):
            assert np.array_equal(x(a), x(b)), n
        ok = np.isfinite(b)
        assert np.isfinite(b[5]).all() and rel_l2(a[ok], b[ok]) < 1e-12, n
