"""The work that users of this library have it do, as cases that can be timed.

A case names one pass through the public classes (`HotPathSimulation` and its
components), the grid, the arithmetic form and the options of the run:

  step        one time step of the hot path, or (physics) of the whole case
              with its surface, forcing, radiation and Smagorinsky terms
  thermo      one thermodynamics update (optionally with the learned seed)
  scalars     the advection tendencies of the scalars
  momentum    the advection tendencies of u, v, w
  pressure    one pressure solve with its ghost fill
  diffusion   Smagorinsky viscosity, scalar and momentum diffusion
  statistics  the horizontal statistics of one output time

`listed()` holds the sizes of this repository's own configurations (32^3 dry,
64x64x75 BOMEX, 256x256x128, 512x512x256 DYCOMS) and ragged ones around them;
`draw()` gives other grids and options of the same ranges.  The states are the
case's profiles with turbulent perturbations drawn on the GPU from the seed.
"""
from __future__ import annotations

import functools
import math

import torch

from pycles_b200 import cases as initial_states
from pycles_b200.grid import Grid
from pycles_b200.learned import cell_inputs, train_seed
from pycles_b200.reference_state import ReferenceState
from pycles_b200.simulation import HotPathSimulation, namelist_for
from pycles_b200.statistics import HorizontalStatistics
from pycles_b200.thermodynamics import ThermodynamicsDry, ThermodynamicsSA

# horizontal spacing, column height, time step and casename of each case
SETUPS = {
    "dry_cbl": dict(dx=50.0, height=1600.0, dt=0.5, casename="SullivanPatton"),
    "bomex": dict(dx=100.0, height=3000.0, dt=1.0, casename="Bomex"),
    "dycoms": dict(dx=35.0, height=1500.0, dt=0.25, casename="DYCOMS_RF01"),
}


def listed():
    return [
        # the smallest whole step: a teaching or test run, bound by launches
        _case("dry_step_32", "step", "dry_cbl", 32, 32, 32, physics=True),
        # the standard BOMEX run as a user steps it, every term of the case on
        _case("bomex_case_64x64x75", "step", "bomex", 64, 64, 75, physics=True),
        # a stratocumulus case run with radiation, WENO7 scalars, and a grid that is no power of two
        _case("dycoms_case_96x96x150", "step", "dycoms", 96, 96, 150, gw=4, order=7, physics=True),
        # the large benchmark step: the dynamical core alone in the precision form
        _case("dycoms_step_512x512x256_fp32", "step", "dycoms", 512, 512, 256, gw=4, order=7, precision="fp32"),
        # saturation adjustment of a cloud-topped state in the plain form
        _case("thermo_256x256x128", "thermo", "dycoms", 256, 256, 128),
        # the same in the precision form with the learned seed for the secant
        _case("thermo_256x256x256_fp32_seed", "thermo", "dycoms", 256, 256, 256, precision="fp32", seeded=True),
        # scalar advection at the 256x256x128 BOMEX size
        _case("scalars_256x256x128", "scalars", "bomex", 256, 256, 128),
        # momentum advection on a ragged grid with an odd number of levels
        _case("momentum_200x180x101", "momentum", "bomex", 200, 180, 101),
        # the pressure solve of the 256x256x128 configuration, plain form
        _case("pressure_256x256x128", "pressure", "bomex", 256, 256, 128),
        # the pressure solve of a grid whose sides are composite numbers, precision form
        _case("pressure_150x120x90_fp32", "pressure", "bomex", 150, 120, 90, precision="fp32"),
        # the subgrid-scale part of a stage
        _case("diffusion_192x192x150", "diffusion", "dycoms", 192, 192, 150),
        # the profiles that a run writes at an output time
        _case("statistics_256x256x128", "statistics", "bomex", 256, 256, 128),
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "thermo", "scalars", "momentum", "pressure", "diffusion", "statistics"])
    setup = rng.choice(["dry_cbl", "bomex", "dycoms", "dycoms"])
    if kind == "thermo" and setup == "bomex":
        setup = "dycoms"
    most = 6.0e6 if kind == "step" else 1.6e7  # cells

    def side():
        if rng.random() < 0.4:
            return rng.choice([32, 64, 128, 256, 512])
        n = int(round(math.exp(rng.uniform(math.log(24), math.log(400)))))
        return n if rng.random() < 0.5 else 2 * (n // 2)

    while True:
        nx, ny = side(), side()
        nz = int(round(math.exp(rng.uniform(math.log(30), math.log(300)))))
        if nx * ny * nz <= most:
            break
    order = rng.choice([5, 5, 7])
    physics = kind == "step" and rng.random() < 0.5
    precision = "fp64" if physics or kind == "diffusion" else rng.choice(["fp64", "fp32"])
    seeded = kind == "thermo" and setup == "dycoms" and precision == "fp32" and rng.random() < 0.5
    return _case(None, kind, setup, nx, ny, nz, gw=4 if order == 7 else 3, order=order, precision=precision,
                 physics=physics, seeded=seeded)


def _case(name, kind, setup, nx, ny, nz, gw=3, order=5, precision="fp64", physics=False, seeded=False):
    c = dict(kind=kind, setup=setup, nx=nx, ny=ny, nz=nz, gw=gw, order=order, precision=precision, physics=physics,
             seeded=seeded)
    return c if name is None else dict(c, name=name)


# ---------------------------------------------------------------------------
# states
# ---------------------------------------------------------------------------
def _namelist(case):
    s = SETUPS[case["setup"]]
    nl = namelist_for(case["setup"], case["nx"], case["ny"], case["nz"], s["dx"], s["dx"], s["height"] / case["nz"],
                      gw=case["gw"], dt=s["dt"], scalar_order=case["order"], momentum_order=5,
                      precision=case["precision"])
    if case["physics"]:
        nl["meta"] = {"casename": s["casename"]}
    if case["physics"] or case["kind"] == "diffusion":
        nl["sgs"] = {"scheme": "Smagorinsky"}
        nl["diffusion"] = {"qt_entropy_source": case["setup"] != "dry_cbl"}
    return nl


@functools.lru_cache(maxsize=64)
def _profiles(setup, nz, gw):
    """The case's reference state and its initial profiles (one column)."""
    s = SETUPS[setup]
    nl = namelist_for(setup, 4, 4, nz, s["dx"], s["dx"], s["height"] / nz, gw=gw)
    Gr = Grid(nl)
    Gr.device = "cpu"
    RS = ReferenceState(Gr)
    Th = ThermodynamicsDry(nl) if setup == "dry_cbl" else ThermodynamicsSA(nl)
    f = initial_states.CASES[setup](Gr, RS, Th, seed=0)
    col = {n: torch.from_numpy(a.reshape(Gr.shape).mean(axis=(0, 1)).copy()) for n, a in f.items()}
    return RS.profiles(), col, torch.from_numpy(Gr.z_half.copy())


def _noise(shape, gen):
    """Random numbers of unit variance, correlated over a few cells."""
    x = torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64) - 0.5
    for d in (0, 1):
        x = x + 0.5 * (torch.roll(x, 1, d) + torch.roll(x, -1, d))
    y = x.clone()
    y[:, :, 1:-1] += 0.5 * (x[:, :, 2:] + x[:, :, :-2])
    return y / y.std()


def prepare(case, seed):
    nl = _namelist(case)
    sim = HotPathSimulation(nl, device="cuda")
    rs, col, z_half = _profiles(case["setup"], case["nz"], case["gw"])
    sim.set_reference_state(rs)
    Gr, PV = sim.Gr, sim.PV
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    height = SETUPS[case["setup"]]["height"]
    z = z_half.cuda()
    # a turbulent layer over the lower two thirds of the column
    env = lambda x: torch.clamp(torch.sin(math.pi * torch.clamp(x / (0.7 * height), 0.0, 1.0)), min=0.0) + 0.02  # noqa: E731
    inner = Gr.interior()
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    for n in PV.index_name:
        a = PV.get_variable_array(n, Gr)
        a.copy_(col[n].cuda().expand(a.shape))
        if n in ("s", "qt"):
            a[inner] += ({"s": 0.25, "qt": 1.0e-4}[n] * env(z[inner[2]])) * _noise((nx, ny, nz), gen)
    # velocities: the curl of a random vector potential on the cell edges, so
    # that the mass flux is free of divergence, as every step leaves it
    dims = Gr.dims
    faces = torch.arange(nz + 1, device="cuda", dtype=torch.float64) * dims.dx[2]
    wall = env(faces)
    wall[0] = wall[-1] = 0.0
    ax, ay = (wall * _noise((nx, ny, nz + 1), gen) for _ in range(2))
    prof = {k: torch.as_tensor(rs[k], device="cuda", dtype=torch.float64) for k in ("rho0", "rho0_half")}
    u, v, w = (PV.get_variable_array(n, Gr)[inner] for n in "uvw")
    du = -(ay[:, :, 1:] - ay[:, :, :-1]) / dims.dx[2]
    scale = 0.5 / du.std()
    u += scale * du / prof["rho0_half"][inner[2]]
    v += scale * (ax[:, :, 1:] - ax[:, :, :-1]) / dims.dx[2] / prof["rho0_half"][inner[2]]
    curl = (ay - torch.roll(ay, 1, 0)) / dims.dx[0] - (ax - torch.roll(ax, 1, 1)) / dims.dx[1]
    w += scale * curl[:, :, 1:] / prof["rho0"][inner[2]]
    if case["kind"] in ("pressure", "statistics"):  # what the advection and the buoyancy of a stage add
        for a in (u, v, w):
            a += 0.01 * env(z[inner[2]]) * _noise((nx, ny, nz), gen)
        w[:, :, -1] = 0.0
    del ax, ay, curl, du
    PV.Update_all_bcs(Gr)
    state = {"case": case, "sim": sim}
    kind = case["kind"]
    if kind in ("diffusion", "statistics"):
        sim.Th.update(Gr, sim.RS, PV, sim.DV)
    if case["seeded"]:
        sim.Th.update(Gr, sim.RS, PV, sim.DV)
        PV.tendencies.zero_()
        sim.Th.mlp, _ = train_seed(sim.Th, [cell_inputs(sim)], n_pairs=200_000, epochs=3, n_held_out=10_000,
                                   draw=2_000_000, max_draws=4)
    if kind == "statistics":
        state["stats"] = HorizontalStatistics(Gr)
        state["mask"] = ((sim.DV.field("ql", Gr) > 0.0) if sim.moist else (PV.field("w", Gr) > 0.0)).double()
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    case, sim = state["case"], state["sim"]
    Gr, PV, DV, RS = sim.Gr, sim.PV, sim.DV, sim.RS
    kind = case["kind"]
    if kind == "step":
        sim.step()
        out = {n: PV.field(n, Gr) for n in PV.index_name}
        out["temperature"] = DV.field("temperature", Gr)
        out["dynamic_pressure"] = DV.field("dynamic_pressure", Gr)
        return out
    if kind == "thermo":
        sim.Th.update(Gr, RS, PV, DV)
        out = {n: DV.field(n, Gr) for n in DV.index_name if n not in ("dynamic_pressure", "divergence")}
        out["w_tendency"] = PV.tendency("w", Gr)
        if sim.moist:
            out["qt"] = PV.field("qt", Gr)
        return out
    if kind == "scalars":
        sim.SA.update(Gr, RS, PV, DV)
        t = PV.tendencies  # (the precision form launches the advection that nothing else takes up here)
        npg = Gr.npg
        return {n: t[PV.get_nv(n) * npg:(PV.get_nv(n) + 1) * npg] for n in PV.index_name if n in ("s", "qt")}
    if kind == "momentum":
        sim.MA.update(Gr, RS, PV)
        t = PV.tendencies
        npg = Gr.npg
        return {n: t[PV.get_nv(n) * npg:(PV.get_nv(n) + 1) * npg] for n in ("u", "v", "w")}
    if kind == "pressure":
        sim.Pr.update(Gr, RS, DV, PV)
        out = {n: PV.field(n, Gr) for n in ("u", "v", "w")}
        out["divergence"] = DV.field("divergence", Gr)
        out["dynamic_pressure"] = DV.field("dynamic_pressure", Gr)
        return out
    if kind == "diffusion":
        sim.SGS.update(Gr, DV, PV, sim.Ke, sim.Sur)
        sim.SD.update(Gr, RS, PV, DV)
        sim.MD.update(Gr, RS, PV, DV, sim.Ke)
        out = {n + "_tendency": PV.tendency(n, Gr) for n in PV.index_name}
        out.update(viscosity=DV.field("viscosity", Gr), diffusivity=DV.field("diffusivity", Gr),
                   strain_rate_mag=sim.Ke.strain_rate_mag)
        return out
    st, mask = state["stats"], state["mask"]
    out = {}
    for n in PV.index_name + ["temperature"]:
        f = DV.field(n, Gr) if n == "temperature" else PV.field(n, Gr)
        out[n + "_mean"] = st.HorizontalMean(Gr, f)
        out[n + "_mean2"] = st.HorizontalMeanofSquares(Gr, f, f)
        out[n + "_max"] = st.HorizontalMaximum(Gr, f)
        out[n + "_min"] = st.HorizontalMinimum(Gr, f)
        out[n + "_conditional"] = st.HorizontalMeanConditional(Gr, f, mask)
    w = PV.field("w", Gr)
    out["w_mean3"] = st.HorizontalMeanofCubes(Gr, w, w, w)
    for n in ("u", "v", "s"):
        out["w" + n] = st.HorizontalMeanofSquares(Gr, w, PV.field(n, Gr))
    return out


def work(case):
    """Each input once, each output once (8-byte values); operations of the
    formulas that have to be evaluated."""
    n = float(case["nx"] * case["ny"] * case["nz"])
    moist = case["setup"] != "dry_cbl"
    ns, nv = (2, 5) if moist else (1, 4)
    weno_s, weno_m = (150.0 if case["order"] == 5 else 302.0), 155.0
    kind = case["kind"]
    thermo_b, thermo_f = (8.0 * 14, 250.0) if moist else (8.0 * 7, 90.0)
    if kind == "thermo":
        return {"bytes": thermo_b * n, "flops": thermo_f * n}
    if kind == "scalars":
        return {"bytes": 8.0 * (3 + 3 * ns) * n, "flops": 3.0 * ns * weno_s * n}
    if kind == "momentum":
        return {"bytes": 8.0 * 9 * n, "flops": 9.0 * weno_m * n}
    fft = 2.5 * 2 * (math.log2(case["nx"]) + math.log2(case["ny"])) + 40.0
    if kind == "pressure":
        return {"bytes": 8.0 * 8 * n, "flops": fft * n}
    diff_b, diff_f = 8.0 * (4 + 3 + 3 * nv + 3), 150.0 + 60.0 * ns + 250.0
    if kind == "diffusion":
        return {"bytes": diff_b * n, "flops": diff_f * n}
    if kind == "statistics":
        return {"bytes": 8.0 * (nv + 2) * n, "flops": 6.0 * (nv + 1) * n}
    # a stage: thermodynamics, advection with the Runge-Kutta update, pressure
    b = thermo_b + 8.0 * 3 * nv + 8.0 * 8
    f = thermo_f + 3.0 * ns * weno_s + 9.0 * weno_m + 4.0 * nv + fft
    if case["physics"]:
        b, f = b + diff_b, f + diff_f
    return {"bytes": 3 * b * n, "flops": 3 * f * n}


# ---------------------------------------------------------------------------
# the same results in plain torch, 64 bits
# ---------------------------------------------------------------------------
G, RD, RV, EPSV, EPSVI = 9.80665, 287.1, 461.5, 0.6221018418201517, 1.6074538488331591
CPD, CPV, KAPPA, T0, P0 = 1004.0, 1859.0, 0.2859561752988048, 298.15, 100000.0
SD0, SV0 = 6864.8, 10513.6


def exact(case, seed):
    """What `run` returns, from plain torch formulas on the same inputs.  The
    whole-case steps (surface, forcing, radiation) have no such value."""
    if case["physics"]:
        return None
    state = prepare(dict(case, seeded=False), seed)
    m = _Exact(case, state)
    kind = case["kind"]
    if kind == "step":
        return m.step()
    if kind == "thermo":
        out = m.thermo()
        out["w_tendency"] = m.t["w"]
        if m.moist:
            out["qt"] = m.f["qt"]
    elif kind == "scalars":
        m.scalars()
        out = {n: m.t[n] for n in ("s", "qt") if n in m.t}
    elif kind == "momentum":
        m.momentum()
        out = {n: m.t[n] for n in ("u", "v", "w")}
    elif kind == "pressure":
        div, p = m.pressure()
        out = {n: m.f[n] for n in ("u", "v", "w")}
        out.update(divergence=div, dynamic_pressure=p)
    elif kind == "diffusion":
        out = m.diffusion()
    else:
        return m.statistics(state["mask"])
    return {n: (a.reshape(-1) if a is not None else None) for n, a in out.items()}


class _Exact:
    def __init__(self, case, state):
        sim = state["sim"]
        self.Gr, d = sim.Gr, sim.Gr.dims
        self.gw, self.n = case["gw"], (case["nx"], case["ny"], case["nz"])
        self.dx = [d.dx[i] for i in range(3)]
        self.moist, self.order, self.dt = sim.moist, case["order"], SETUPS[case["setup"]]["dt"]
        self.f = {n: sim.PV.get_variable_array(n, sim.Gr).clone() for n in sim.PV.index_name}
        self.t = {n: torch.zeros_like(a) for n, a in self.f.items()}
        if case["kind"] in ("diffusion", "statistics"):
            self.t["w"] = sim.PV.get_tendency_array("w", sim.Gr).clone()  # the buoyancy of prepare()'s update
        for k in ("p0_half", "alpha0", "alpha0_half", "rho0", "rho0_half"):
            setattr(self, k, torch.as_tensor(getattr(sim.RS, k), device="cuda", dtype=torch.float64))
        cc = sim.Th.CC
        self.table = torch.as_tensor(cc.pv, device="cuda", dtype=torch.float64)
        self.tab = (cc.x_min, cc.dx, cc.dxi)
        self.inner = sim.Gr.interior()
        self.dv = {n: sim.DV.get_variable_array(n, sim.Gr) for n in sim.DV.index_name}

    # ghosts: periodic in x and y, mirrored (sym) or odd (asym) in z
    def ghosts(self, a, sym=True):
        g = self.gw
        a[:g] = a[-2 * g:-g].clone()
        a[-g:] = a[g:2 * g].clone()
        a[:, :g] = a[:, -2 * g:-g].clone()
        a[:, -g:] = a[:, g:2 * g].clone()
        n = a.shape[2]
        for q in range(g):
            if sym:
                a[:, :, n - g + q] = a[:, :, n - g - 1 - q]
                a[:, :, g - 1 - q] = a[:, :, g + q]
            else:
                a[:, :, n - g + q] = 0.0 if q == 0 else -a[:, :, n - g - q]
                a[:, :, g - 1 - q] = 0.0 if q == 0 else -a[:, :, g - 1 + q]

    # thermodynamics ---------------------------------------------------------
    def lookup(self, x):
        x_min, dx, dxi = self.tab
        fi = torch.floor((x - x_min) * dxi).clamp(0, self.table.numel() - 2)
        i = fi.long()
        y1, y2 = self.table[i], self.table[i + 1]
        return y1 + (x - (x_min + dx * fi)) * (y2 - y1) * dxi

    @staticmethod
    def latent(T):
        c = T - 273.15
        return (2500.8 - 2.36 * c + 0.0016 * c * c - 0.00006 * c * c * c) * 1000.0

    @staticmethod
    def entropy(pd, pv, T, qt, L, sig):
        return ((SD0 + CPD * torch.log(T / T0) - RD * torch.log(pd / P0)) * (1.0 - qt)
                + (SV0 + CPV * torch.log(T / T0) - RV * torch.log(pv / P0)) * qt - L / T * sig)

    def eos(self, p0, s, qt):
        """The saturation adjustment's secant, to 1e-3 K."""
        pv = p0 * EPSVI * qt / (1.0 - qt + EPSVI * qt)
        pd = p0 - pv
        T1 = T0 * torch.exp((s - (1.0 - qt) * (SD0 - RD * torch.log(pd / P0)) - qt * (SV0 - RV * torch.log(pv / P0)))
                            / ((1.0 - qt) * CPD + qt * CPV))
        pvs = self.lookup(T1)
        qs = EPSV * (1.0 - qt) * pvs / (p0 - pvs)
        T, ql = T1.clone(), torch.zeros_like(T1)
        at = torch.nonzero((qt > qs).reshape(-1)).reshape(-1)
        if at.numel():
            pick = lambda a: a.reshape(-1)[at]  # noqa: E731
            P, S, Q, t1, q1 = pick(p0.expand(s.shape)), pick(s), pick(qt), pick(T1), pick(qs)
            sig = Q - q1
            L = self.latent(t1)
            f1 = S - self.entropy(pick(pd), pick(pv), t1, Q, L, sig)
            t2 = t1 + sig * L / ((1.0 - Q) * CPD + q1 * CPV)
            out_t, out_q = t2.clone(), sig.clone()
            act = torch.arange(at.numel(), device=at.device)
            for _ in range(100):
                if not act.numel():
                    break
                pvs = self.lookup(t2)
                qs = EPSV * (1.0 - Q) * pvs / (P - pvs)
                pv2 = P * EPSVI * qs / (1.0 - Q + EPSVI * qs)
                sig = Q - qs
                f2 = S - self.entropy(P - pv2, pv2, t2, Q, self.latent(t2), sig)
                tn = t2 - f2 * (t2 - t1) / (f2 - f1)
                out_t[act], out_q[act] = tn, sig
                more = ((tn - t2).abs() >= 1.0e-3) | (sig < 0.0)
                act, P, S, Q = act[more], P[more], S[more], Q[more]
                t1, t2, f1 = t2[more], tn[more], f2[more]
            T.view(-1)[at] = out_t
            ql.view(-1)[at] = out_q
        return T, ql

    def thermo(self):
        p0, a0, n = self.p0_half, self.alpha0_half, self.p0_half.numel()
        ex = (p0 / P0) ** KAPPA
        dzi = 1.0 / self.dx[2]
        wt, s = self.t["w"], self.f["s"]
        mid = lambda a, b: 0.5 * (a + b)  # noqa: E731
        if not self.moist:
            T = T0 * torch.exp((s - SD0 + RD * torch.log(p0 / P0)) / CPD)
            al = RD * T / p0
            b = torch.zeros_like(T)
            b[:-1, :-1, :-1] = (G * (al - a0) / a0)[:-1, :-1, :-1]
            wt[:-1, :-1, :-1] += mid(b[:-1, :-1, :-1], b[:-1, :-1, 1:])
            th = torch.zeros_like(T)
            th[:, :, 1:] = (T / ex)[:, :, 1:]
            bv = torch.zeros_like(T)
            bv[:, :, 2:n - 1] = G / th[:, :, 2:n - 1] * (th[:, :, 3:] - th[:, :, 1:n - 2]) * 0.5 * dzi
            return dict(temperature=T, alpha=al, buoyancy=b, theta=th, buoyancy_frequency=bv)
        qt = self.f["qt"]
        qt.clamp_(min=1e-11)
        T, ql = self.eos(p0, s, qt)
        qv = qt - ql
        al = RD * T / p0 * (1.0 - qt + EPSVI * qv)
        b = torch.zeros_like(T)
        b[:, :, :-1] = (G * (al - a0) / a0)[:, :, :-1]
        wt[:, :, 1:n - 3] += mid(b[:, :, 1:n - 3], b[:, :, 2:n - 2])
        thr = torch.zeros_like(T)
        thr[:, :, 1:-1] = (T * (1.0 - qt + EPSVI * qv) / ex)[:, :, 1:-1]
        k, up, dn = slice(2, n - 2), slice(3, n - 1), slice(1, n - 3)
        Tk, Qk, Pk = T[:, :, k], qt[:, :, k], p0[k]
        L, pvs = self.latent(Tk), self.lookup(Tk)
        r = EPSV * pvs / (Pk - pvs)
        gam = (G / CPD * (1.0 / (1.0 - Qk)) * (1.0 + L * r / (RD * Tk))
               / (((1.0 - Qk) * CPD + Qk * CPV) / CPD + L * L * (EPSV + r) * r / (CPD * RD * Tk * Tk)))
        grad = lambda a: (a[:, :, up] - a[:, :, dn]) * 0.5 * dzi  # noqa: E731
        wet = G / Tk * (grad(T) + gam) * (1.0 + L * r / (RD * Tk)) - grad(qt) / (1.0 - Qk)
        bv = torch.zeros_like(T)
        bv[:, :, k] = torch.where(ql[:, :, k] > 0.0, wet, G / thr[:, :, k] * grad(thr))
        thl = T / ex * torch.exp(-self.latent(T) * (ql / (1.0 - qt)) / (T * CPD))
        return dict(temperature=T, qv=qv, ql=ql, qi=torch.zeros_like(ql), alpha=al, buoyancy=b, theta_rho=thr,
                    buoyancy_frequency=bv, thetali=thl)

    # advection ----------------------------------------------------------------
    @staticmethod
    def weno(v):
        if len(v) == 5:
            a, b, c, d, e = v
            p = (a / 3 - 7 / 6 * b + 11 / 6 * c, -b / 6 + 5 / 6 * c + d / 3, c / 3 + 5 / 6 * d - e / 6)
            q = (13 / 12 * (a - 2 * b + c) ** 2 + (a - 4 * b + 3 * c) ** 2 / 4,
                 13 / 12 * (b - 2 * c + d) ** 2 + (b - d) ** 2 / 4,
                 13 / 12 * (c - 2 * d + e) ** 2 + (3 * c - 4 * d + e) ** 2 / 4)
            lin = (0.1, 0.6, 0.3)
            centre = 0.0
        else:
            centre = v[3]
            a, b, c, d, e, f, g = (x - centre for x in v)  # (the indicators cancel: on differences)
            p = (-a / 4 + 13 / 12 * b - 23 / 12 * c + 25 / 12 * d, b / 12 - 5 / 12 * c + 13 / 12 * d + e / 4,
                 -c / 12 + 7 / 12 * d + 7 / 12 * e - f / 12, d / 4 + 13 / 12 * e - 5 / 12 * f + g / 12)
            q = (a * (547 * a - 3882 * b + 4642 * c - 1854 * d) + b * (7043 * b - 17246 * c + 7042 * d)
                 + c * (11003 * c - 9402 * d) + 2107 * d * d,
                 b * (267 * b - 1642 * c + 1602 * d - 494 * e) + c * (2843 * c - 5966 * d + 1922 * e)
                 + d * (3443 * d - 2522 * e) + 547 * e * e,
                 c * (547 * c - 2522 * d + 1922 * e - 494 * f) + d * (3443 * d - 5966 * e + 1602 * f)
                 + e * (2843 * e - 1642 * f) + 267 * f * f,
                 d * (2107 * d - 9402 * e + 7042 * f - 1854 * g) + e * (11003 * e - 17246 * f + 4642 * g)
                 + f * (7043 * f - 3882 * g) + 547 * g * g)
            lin = (1 / 35, 12 / 35, 18 / 35, 4 / 35)
        w = [c_ / (q_ + 1e-10) ** 2 for c_, q_ in zip(lin, q)]
        return centre + sum(w_ * p_ for w_, p_ in zip(w, p)) / sum(w)

    def at(self, a, axis, o, other=None, oo=0):
        """`a` on the faces of `axis` (lower cells gw-1 .. n-gw-1; interior
        elsewhere), moved by o along axis (and by oo along `other`)."""
        g, ix = self.gw, []
        for d in range(3):
            lo, hi = g - (1 if d == axis else 0), g + self.n[d]
            m = (o if d == axis else 0) + (oo if d == other else 0)
            ix.append(slice(lo + m, hi + m))
        return a[tuple(ix)]

    def face(self, a, vel, axis, order):
        r = order // 2
        up = self.weno([self.at(a, axis, o) for o in range(-r, r + 1)])
        dn = self.weno([self.at(a, axis, o) for o in range(r + 1, -r, -1)])
        return torch.where(vel >= 0.0, up, dn) * vel

    def level(self, prof, axis, o=0):
        g = self.gw
        return prof[g - (1 if axis == 2 else 0) + o:g + self.n[2] + o]

    @staticmethod
    def diff(F, axis):
        m = F.shape[axis]
        return F.narrow(axis, 1, m - 1) - F.narrow(axis, 0, m - 1)

    def scalars(self):
        al = self.alpha0_half[self.inner[2]]
        for n in ("s", "qt"):
            if n not in self.f:
                continue
            for d, v in enumerate("uvw"):
                F = self.face(self.f[n], self.at(self.f[v], d, 0), d, self.order)
                F = F * self.level(self.rho0 if d == 2 else self.rho0_half, d)
                self.t[n][self.inner] -= al * self.diff(F, d) / self.dx[d]

    def momentum(self):
        for c, n in enumerate("uvw"):
            al = (self.alpha0 if c == 2 else self.alpha0_half)[self.inner[2]]
            for d, v in enumerate("uvw"):
                a = self.f[v]
                x = [self.at(a, d, o) if c == d else self.at(a, d, 0, c, o) for o in (-1, 0, 1, 2)]
                vel = 7 / 12 * (x[1] + x[2]) - (x[0] + x[3]) / 12
                F = self.face(self.f[n], vel, d, 5)
                if c == 2 and d == 2:
                    F = F * self.level(self.rho0_half, d, 1)
                else:
                    F = F * self.level(self.rho0 if 2 in (c, d) else self.rho0_half, d)
                self.t[n][self.inner] -= al * self.diff(F, d) / self.dx[d]

    # pressure -------------------------------------------------------------------
    def pressure(self):
        g, (nx, ny, nz), dx = self.gw, self.n, self.dx
        f, I = self.f, self.inner
        f["w"] -= f["w"][I[0], I[1]].mean(dim=(0, 1))
        k = I[2]
        U, V, W = f["u"], f["v"], f["w"]
        lower = lambda a, d: a[tuple(slice(s.start - (q == d), s.stop - (q == d)) for q, s in enumerate(I))]  # noqa: E731
        dn = slice(k.start - 1, k.stop - 1)
        rhs = ((U[I] - lower(U, 0)) / dx[0] + (V[I] - lower(V, 1)) / dx[1]) / self.alpha0_half[k]
        rhs += (W[I] / self.alpha0[k] - lower(W, 2) / self.alpha0[dn]) / dx[2]
        div = torch.zeros_like(U)
        div[I] = rhs
        wave = lambda n, h: (2.0 * torch.cos(2.0 * math.pi / n * torch.arange(n, device="cuda", dtype=torch.float64))  # noqa: E731
                             - 2.0) / (h * h)
        kk = wave(nx, dx[0])[:, None] + wave(ny, dx[1])[None, :]
        X = torch.fft.fft2(rhs, dim=(0, 1)).permute(2, 0, 1).contiguous()
        iz2 = 1.0 / dx[2] ** 2
        r0, rh = (self.rho0 * iz2).tolist(), self.rho0_half.tolist()
        c, prev = torch.empty((nz, nx, ny), device="cuda", dtype=torch.float64), None
        kk[0, 0] = -1.0  # (its column is set to zero)
        for q in range(nz):
            lo, hi = (r0[q + g - 1] if q > 0 else 0.0), (r0[q + g] if q < nz - 1 else 0.0)
            b = rh[q + g] * kk - (lo + hi)
            m = 1.0 / (b - lo * c[q - 1]) if q > 0 else 1.0 / b
            c[q] = hi * m
            X[q] = (X[q] - lo * X[q - 1]) * m if q > 0 else X[q] * m
        for q in range(nz - 2, -1, -1):
            X[q] -= c[q] * X[q + 1]
        X[:, 0, 0] = 0.0
        p = torch.zeros_like(U)
        p[I] = torch.fft.ifft2(X, dim=(1, 2)).real.permute(1, 2, 0)
        self.ghosts(p)
        for d, n in enumerate("uvw"):
            cut = tuple(slice(0, s - 1) for s in p.shape)
            f[n][cut] -= self.diff(p, d)[tuple(slice(0, s - 1) for s in p.shape)] / dx[d]
        for n in "uvw":
            self.ghosts(f[n], n != "w")
        return div, p

    def step(self):
        copy = {n: a.clone() for n, a in self.f.items()}
        for a, b in ((0.0, 1.0), (0.75, 0.25), (1 / 3, 2 / 3)):
            T = self.thermo()["temperature"]
            self.scalars()
            self.momentum()
            for n in self.f:
                self.f[n] = a * copy[n] + b * (self.f[n] + self.t[n] * self.dt)
                self.t[n].zero_()
                self.ghosts(self.f[n], n != "w")
            _, p = self.pressure()
        out = {n: v.reshape(-1) for n, v in self.f.items()}
        out.update(temperature=T.reshape(-1), dynamic_pressure=p.reshape(-1))
        return out

    # subgrid scale ----------------------------------------------------------------
    def diffusion(self):
        f, dx, I = self.f, self.dx, self.inner
        vel = [f[n] for n in "uvw"]
        sh = lambda a, d, o: torch.roll(a, -o, d)  # noqa: E731  (wraps only where no interior cell reads)
        S = {}
        for a in range(3):
            for b in range(3):
                S[a, b] = 0.5 * ((sh(vel[a], b, 1) - vel[a]) / dx[b] + (sh(vel[b], a, 1) - vel[b]) / dx[a])
        m = sum(sh(S[d, d], d, -1) ** 2 for d in range(3))
        for a, b in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2)):
            s = S[a, b]
            m = m + 2.0 * (0.25 * (s + sh(s, a, -1) + sh(s, b, -1) + sh(sh(s, a, -1), b, -1))) ** 2
        mag = torch.sqrt(2.0 * m)
        cs, prt = 0.17, 1.0 / 3.0
        nu = (cs * (dx[0] * dx[1] * dx[2]) ** (1.0 / 3.0)) ** 2 * mag
        n2 = self.dv["buoyancy_frequency"]
        nu = torch.where(n2 > 0.0, nu * torch.sqrt(torch.clamp(1.0 - n2 / (prt * mag * mag), min=0.0)), nu)
        D = nu / prt
        T = self.dv["temperature"]
        kz = torch.arange(T.shape[2], device="cuda")
        below = kz == self.gw - 1
        for n in ("s", "qt"):
            if n not in f:
                continue
            if n == "qt":
                qt, qv = f["qt"], self.dv["qv"]
                den = 1.0 - qt + EPSVI * qv
                sd = SD0 + CPD * torch.log(T / T0) - RD * torch.log(self.p0_half * (1.0 - qt) / den / P0)
                sv = SV0 + CPV * torch.log(T / T0) - RV * torch.log(self.p0_half * EPSVI * qv / den / P0)
                src = sv - (qt - qv) / qt * self.latent(T) / T - sd
            for d in range(3):
                F = -0.5 * (D + sh(D, d, 1)) * (sh(f[n], d, 1) - f[n]) / dx[d]
                F = F * (self.rho0 if d == 2 else self.rho0_half)
                F = torch.where(below, torch.zeros_like(F), F)
                self.t[n][I] -= (self.alpha0_half * (F - sh(F, d, -1)) / dx[d])[I]
                if n == "qt":
                    up = sh(F, d, 1).clone()
                    edge = [slice(None)] * 3
                    edge[d] = I[d].stop - 1  # the face above the last cell is not in the flux's range
                    up[tuple(edge)] = 0.0
                    self.t["s"][I] -= (src * self.alpha0_half * (up - F) / dx[d])[I]
        for a in range(3):
            al = self.alpha0 if a == 2 else self.alpha0_half
            for b in range(3):
                if a == b:
                    v = sh(nu, a, 1)
                    rho = sh(self.rho0_half, 0, 1) if a == 2 else self.rho0_half
                else:
                    v = 0.25 * (nu + sh(nu, a, 1) + sh(nu, b, 1) + sh(sh(nu, a, 1), b, 1))
                    rho = self.rho0 if 2 in (a, b) else self.rho0_half
                F = -2.0 * S[a, b] * v * rho
                F = torch.where(below, torch.zeros_like(F), F)
                self.t["uvw"[a]][I] -= (al * (F - sh(F, b, -1)) / dx[b])[I]
        self.t["s"][I] += (mag * mag * nu / T)[I]
        out = {n + "_tendency": a for n, a in self.t.items()}
        # (the ghost planes of these three follow no formula)
        out.update(viscosity=None, diffusivity=None, strain_rate_mag=None)
        return out

    def statistics(self, mask):
        I = self.inner
        flat = lambda a: a[I[0], I[1]].reshape(-1, a.shape[2])  # noqa: E731
        mk = flat(mask.view(self.f["u"].shape))
        out = {}
        for n in list(self.f) + ["temperature"]:
            a = flat(self.dv[n] if n == "temperature" else self.f[n])
            out[n + "_mean"] = a.mean(dim=0)
            out[n + "_mean2"] = (a * a).mean(dim=0)
            out[n + "_max"], out[n + "_min"] = a.max(dim=0).values, a.min(dim=0).values
            out[n + "_conditional"] = (a * mk).sum(dim=0) / mk.sum(dim=0).clamp(min=1.0)
        w = flat(self.f["w"])
        out["w_mean3"] = (w * w * w).mean(dim=0)
        for n in ("u", "v", "s"):
            out["w" + n] = (w * flat(self.f[n])).mean(dim=0)
        return out
