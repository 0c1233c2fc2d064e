"""Performance cases of the implicit stepping path.

Each case is one call (or the pair of calls that always go together) that a program using this package
makes on its way through a cycle step: the residual and the stage residual, the finite-difference Jacobian,
the preconditioner's factorisation and solve, one implicit stage, a whole integration, a whole cycle step
through the step runner, and the predictor network's training.  Sizes run from the 1x1x30 bed of the 1-D
cases to the 16x16x64 bed of the large cycle; 8x8x12 is the default grid, 8x8x32 the cycle benchmark's.

Beds are drawn from the seed: an adsorption front somewhere in the bed (or a heated bed under vacuum), with
cell-to-cell noise, at the operating point of the cycle benchmark.
"""
from __future__ import annotations

import numpy as np
import torch

from dac_vtsa_b200 import host
from dac_vtsa_b200.config import load_config
from dac_vtsa_b200.runner import BENCH_POINT

STEPS = {"adsorption": 0, "blowdown": 1, "heating": 2, "cooling": 3}


def listed():
    return [
        # latency: one right-hand side of the 1-D bed, the smallest call a driver makes
        {"name": "rhs_1x1x30", "kind": "rhs", "Nr": 1, "Nth": 1, "Nz": 30, "step": "adsorption", "acc": False},
        # right-hand side with the 36 accumulator rates, as each accepted step evaluates it
        {"name": "rhs_acc_8x8x32", "kind": "rhs", "Nr": 8, "Nth": 8, "Nz": 32, "step": "adsorption", "acc": True},
        # Newton residual of an implicit stage on the large bed
        {"name": "stage_16x16x64", "kind": "stage", "Nr": 16, "Nth": 16, "Nz": 64, "step": "heating"},
        # coloured finite-difference Jacobian, refreshed every few dozen steps, ordinary and large bed
        {"name": "jacobian_8x8x32", "kind": "jacobian", "Nr": 8, "Nth": 8, "Nz": 32, "step": "adsorption"},
        {"name": "jacobian_16x16x64", "kind": "jacobian", "Nr": 16, "Nth": 16, "Nz": 64, "step": "heating"},
        # factorisation of I - dh J and one solve with it: what a step-size change costs
        {"name": "factor_8x8x32", "kind": "factor", "Nr": 8, "Nth": 8, "Nz": 32, "step": "adsorption", "dh": 3.0,
         "precision": "fp64", "mode": "theta_block"},
        # one preconditioner solve with factors larger than L2: every Krylov step makes one
        {"name": "solve_16x16x64", "kind": "solve", "Nr": 16, "Nth": 16, "Nz": 64, "step": "heating", "dh": 3.0,
         "precision": "fp64", "mode": "theta_block"},
        # one implicit stage by Newton-Krylov with the factors in hand
        {"name": "newton_8x8x32", "kind": "newton", "Nr": 8, "Nth": 8, "Nz": 32, "step": "adsorption", "dh": 3.0},
        # device-resident integration of a heating window (TR-BDF2), the cycle benchmark's inner loop
        {"name": "heating_8x8x32", "kind": "integrate", "Nr": 8, "Nth": 8, "Nz": 32, "step": "heating",
         "duration": 600.0, "scheme": "trbdf2", "precision": "fp64", "projection": False},
        # a whole blowdown through the step runner at the default grid and scheme: host state in and out,
        # model and integrator built, outlet recorded
        {"name": "blowdown_8x8x12", "kind": "step", "Nr": 8, "Nth": 8, "Nz": 12, "step": "blowdown",
         "duration": 60.0, "scheme": "sdirk2", "spacing": "uniform"},
        # the large bed: adsorption from a fresh front, with the balance projection its cycles run with
        {"name": "adsorption_16x16x64", "kind": "integrate", "Nr": 16, "Nth": 16, "Nz": 64, "step": "adsorption",
         "duration": 20.0, "scheme": "trbdf2", "precision": "fp64", "projection": True},
        # training of the predictor network on samples recorded by the plain solver
        {"name": "train_200", "kind": "train", "Nr": 8, "Nth": 8, "Nz": 12, "step": "heating", "epochs": 200},
    ]


def draw(rng):
    kind = rng.choice(("rhs", "rhs", "stage", "jacobian", "jacobian", "factor", "solve", "solve", "newton",
                       "integrate", "integrate", "step"))

    def log_int(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    while True:
        Nr, Nth, Nz = log_int(1, 16), rng.choice((1, 3, 4, 5, 6, 8, 9, 12, 16)), log_int(6, 64)
        cells = Nr * Nth * Nz
        # whole integrations are kept to beds that the listed ones bound; the rest up to the large bed
        if cells <= (2048 if kind in ("integrate", "step", "newton") else 16384) and (Nr > 1 or Nth == 1):
            break
    c = {"kind": kind, "Nr": Nr, "Nth": Nth, "Nz": Nz, "step": rng.choice(("adsorption", "heating", "cooling"))}
    if kind == "rhs":
        c["acc"] = rng.random() < 0.5
    if kind in ("factor", "solve"):
        c["dh"] = round(0.1 * 300.0 ** rng.random(), 3)
        c["precision"] = rng.choice(("fp64", "fp64", "fp32_factors"))
        c["mode"] = rng.choice(("theta_block", "theta_block", "sector"))
    if kind == "newton":
        c["dh"] = round(0.3 * 30.0 ** rng.random(), 3)
    if kind == "integrate":
        c.update(duration=round(rng.uniform(20.0, 120.0), 1), scheme=rng.choice(("trbdf2", "sdirk2")),
                 precision=rng.choice(("fp64", "fp64", "fp32_factors")), projection=rng.random() < 0.5)
    if kind == "step":
        c.update(step=rng.choice(("blowdown", "cooling")), duration=round(rng.uniform(10.0, 60.0), 1),
                 scheme=rng.choice(("trbdf2", "sdirk2")), spacing=rng.choice(("uniform", "equal_area")))
    return c


# ---------------------------------------------------------------------------- inputs
def _bed(case, seed):
    """Configuration, grid, gas data, cycle step and a drawn bed state of a case."""
    over = dict(BENCH_POINT)
    over.update({"grid.Nr": case["Nr"], "grid.Ntheta": case["Nth"], "grid.Nz": case["Nz"],
                 "solver.scheme": case.get("scheme", "trbdf2"),
                 "grid.radial_spacing": case.get("spacing", "uniform"),
                 "gpu.krylov_precision": case.get("precision", "fp64"),
                 "gpu.balance_projection": bool(case.get("projection", False))})
    cfg = load_config(override_dict=over)
    g = host.Grid.from_config(cfg)
    props = host.get_backend(cfg)
    step = dict(cfg.cycle[STEPS[case["step"]]])
    if "duration" in case:
        step["duration"] = float(case["duration"])
    st = host.initial_state(cfg, g, props)
    rng = np.random.default_rng(seed)
    z = (g.z_c / g.L)[None, None, :]
    r = (g.r_c / g.R)[:, None, None]
    noise = 2.0 * rng.random(g.shape) - 1.0
    zf, width = rng.uniform(0.3, 0.8), rng.uniform(0.06, 0.15)
    behind = 1.0 / (1.0 + np.exp((z + 0.05 * r - zf) / width)) * np.ones(g.shape)   # 1 behind the front
    hot = case["step"] in ("heating", "cooling")
    if hot:          # part-way through desorption: warm bed, water and CO2 under the product vacuum
        T = 318.0 + 30.0 * r ** 2 + 6.0 * z + 0.5 * noise
        y = np.array([0.2, 0.78, 0.02])[:, None, None, None] * np.ones((1,) + g.shape)
        P = 1.02 * cfg.operation.P_vacuum
        q = [0.5 + 0.9 * r + 0.3 * behind, 1.2 + 1.5 * behind]
        Tw = 360.0
    else:            # loaded behind the front, depleted feed ahead of it, the sorption heat at the front
        T = 288.0 + 6.0 * behind * (1.0 - behind) * 4.0 + 0.3 * noise
        y = st.c / st.c.sum(axis=0)
        y = y.copy()
        y[0] *= 0.02 + 0.98 * behind
        y[2] = 1.0 - y[0] - y[1]
        P = 101325.0
        q = [0.05 + 1.3 * behind, 1.5 + 1.7 * behind]
        Tw = 288.0
    st.T = T * np.ones(g.shape)
    st.c = y * (P / (host.R_GAS * st.T))[None]
    st.q = np.stack([a * np.ones(g.shape) * (1.0 + 0.01 * noise) for a in q])
    st.Tw = np.full(g.wall_shape, Tw) + 0.2 * (2.0 * rng.random(g.wall_shape) - 1.0)
    return cfg, g, props, step, st


def prepare(case, seed):
    from dac_vtsa_b200.jacobian import FDJacobian
    from dac_vtsa_b200.model import TVSAModel
    from dac_vtsa_b200.solver import TRBDF2
    cfg, g, props, step, st = _bed(case, seed)
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "step":
        s.update(cfg=cfg, grid=g, props=props, step=step, state=st)
        return s
    m = TVSAModel(cfg, g, props, step, st)
    y = torch.from_numpy(m.pack(st)).to(m.device)
    s.update(m=m, y=y)
    if kind == "stage":
        s["known"] = y * (1.0 + 1e-4)
    if kind in ("jacobian", "factor", "solve", "newton"):
        s["jac"] = FDJacobian(m)
    if kind in ("factor", "solve", "newton"):
        s["J"] = s["jac"].block(1.0, y).clone()
        m.set_krylov_precision(case.get("precision", "fp64"))
        m.precond_factor(s["J"], case["dh"], case.get("mode", "theta_block"))
        # a right-hand side with the distribution of a Newton residual: error scale times noise
        gen = torch.Generator(device="cpu").manual_seed(seed)
        scale = torch.from_numpy(m.atol).to(m.device) + cfg.solver.rtol * y.abs()
        s["b"] = scale * torch.randn(m.n_core, generator=gen, dtype=torch.float64).to(m.device)
    if kind == "integrate":
        s["integ"] = TRBDF2(m, cfg, h_max=cfg.solver.h_max_fraction * step["duration"])
        s["duration"] = step["duration"]
    if kind == "train":
        from dac_vtsa_b200.predictor import NewtonPredictor
        net = NewtonPredictor(sample_capacity=65536, seed=seed)
        integ = TRBDF2(m, cfg, h_max=20.0)
        net.attach(integ, step["type"], predict=False, record_stride=3)
        integ.integrate(y, 20.0, np.array([20.0]), keep_on_device=True)
        P, norm = net.params()
        s.update(net=net, integ=integ, params=P, norm=norm, seed=seed)
    return s


# ---------------------------------------------------------------------------- one pass
def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "rhs":
        f, acc = s["m"].rhs(1.0, s["y"], want_acc=case["acc"])
        return {"f": f, "acc": acc}
    if kind == "stage":
        return {"R": s["m"].stage_residual(1.0, s["y"], 2.0, s["known"])}
    if kind == "jacobian":
        return {"J": s["jac"].block(1.0, s["y"])}
    if kind == "factor":
        s["m"].precond_factor(s["J"], case["dh"], case["mode"])
        return {"x": s["m"].precond_solve(s["b"])}
    if kind == "solve":
        return {"x": s["m"].precond_solve(s["b"])}
    if kind == "newton":
        z, ok, iters, _, stats = s["m"].newton_stage(1.0 + case["dh"], s["y"], s["y"], case["dh"])
        return {"z": z, "ok": ok, "iters": iters, "gmres": int(stats["gmres_iters"])}
    if kind == "integrate":
        d = s["duration"]
        res = s["integ"].integrate(s["y"], d, np.array([d]), keep_on_device=True)
        return {"y": res.y, "acc": res.acc, "steps": int(res.n_steps), "rejected": int(res.n_reject)}
    if kind == "step":
        from dac_vtsa_b200.runner import run_step
        st, sr = run_step(s["state"], s["cfg"], s["grid"], s["props"], s["step"])
        # (the outlet's series has a row per accepted step: its last one, which holds the sums, has a fixed shape)
        keys = [k for k, v in sr.outlet[-1].items() if isinstance(v, float)]
        return {"c": st.c, "q": st.q, "T": st.T, "Tw": st.Tw, "acc": np.array(list(sr.acc.values())),
                "outlet": np.array([sr.outlet[-1][k] for k in keys]), "steps": int(sr.solver["steps"])}
    net = s["net"]
    net.set_params(s["params"], s["norm"])
    loss = net.train(case["epochs"], lr=1e-3, seed=s["seed"])
    P, _ = net.params()
    return {"params": P, "loss": loss}


# ---------------------------------------------------------------------------- floors
def _sizes(case):
    cells = case["Nr"] * case["Nth"] * case["Nz"]
    n = 6 * cells + case["Nth"] * case["Nz"]
    # unknowns of one plane of a preconditioner partition: a sector's rings and its wall node
    nb = min(6 * case["Nr"] + 1, 48) if case["Nth"] > 1 else 6 * case["Nr"] + 1
    blocks = -(-n // nb)                             # planes times partitions
    return cells, n, nb, blocks


def work(case):
    """Bytes: each input read once and each output written once (factors count as an input of a solve).
    Flops: per cell 600 for its closures and fluxes (a transcendental counted as 20), 5 block products and
    an inverse per factorised block, one multiply-add per factor entry in a solve."""
    cells, n, nb, blocks = _sizes(case)
    kind = case["kind"]
    res = 600 * cells
    fac, sol = blocks * 10.0 * nb ** 3, blocks * 10.0 * nb ** 2
    size = 4 if case.get("precision") == "fp32_factors" else 8
    if kind in ("rhs", "stage"):
        return {"bytes": 8 * n * (3 if kind == "stage" else 2), "flops": res}
    if kind == "jacobian":
        # every cell's six perturbations: its closures again, and the faces and balances they reach
        return {"bytes": 8 * (n + 9 * 49 * cells), "flops": 6 * 3 * res}
    if kind == "factor":
        return {"bytes": 8 * (9 * 49 * cells + 2 * n) + size * 5 * blocks * nb ** 2, "flops": fac + sol}
    if kind == "solve":
        return {"bytes": size * 5 * blocks * nb ** 2 + 16 * n, "flops": sol}
    if kind == "train":
        per = 4096 * (112 * 128 + 2 * 128 * 128 + 128 * 16)
        return {"bytes": 4 * 49552 * 2 + 65536 * (224 + 32), "flops": 6.0 * case["epochs"] * per}
    # a stage: at least two Newton iterations of two Krylov steps, each a solve and a residual
    stage_b, stage_f = 4 * (size * 5 * blocks * nb ** 2 + 32 * n), 4 * (sol + res)
    if kind == "newton":
        return {"bytes": stage_b, "flops": stage_f}
    steps = 50 + case["duration"] / (0.02 * case["duration"])    # ramp-up, then the largest step allowed
    return {"bytes": 2 * steps * stage_b, "flops": 2 * steps * stage_f + 2 * fac}


# ---------------------------------------------------------------------------- 64-bit values
def exact(case, seed):
    """Residual and Jacobian by numpy in 64 bits (an integration, a stage and a solve depend on the
    Jacobian's difference quotients and on step control: no value of their own)."""
    kind = case["kind"]
    if kind not in ("rhs", "stage", "jacobian") or (kind == "jacobian" and case["Nr"] * case["Nth"] * case["Nz"] > 2048):
        return None
    cfg, g, props, step, st = _bed(case, seed)
    R = _Residual(cfg, g, props, step, st)
    y = R.pack(st)
    if kind == "rhs":
        return {"f": R(1.0, y), "acc": None}
    if kind == "stage":
        return {"R": y - 2.0 * R(1.0, y) - y * (1.0 + 1e-4)}
    return {"J": R.jacobian(1.0, y)}


class _Residual:
    """dy/dt of the bed at the closures these cases run with (WADST co-adsorption, Edwards-Richardson
    dispersion, Zehner-Schluender conductivity, Martin-Nilles wall, van Albada slopes)."""

    def __init__(self, cfg, g, props, step, st):
        self.cfg, self.g, self.props, self.step = cfg, g, props, step
        self.cond = host.end_conditions(cfg, step, list(props.species), props)
        self.P0 = {"top": st.P[:, :, 0].mean(), "bottom": st.P[:, :, -1].mean()}
        prof = host.feed_profile(cfg, g)
        feed = any(c.kind == "feed" for c in self.cond.values())
        self.Fin = host.feed_molar_flux(cfg) * prof * g.Az
        self.Nnom = (host.feed_molar_flux(cfg) * prof if feed else np.zeros((g.Nr, g.Nth)))[:, :, None]
        self.unom = cfg.feed.velocity if feed else 0.0
        self.cov = g.coverage_fraction(cfg.jacket.theta_coverage_deg, cfg.jacket.z_coverage)

    def _heat(self, c, q):
        so, th, d = self.cfg.sorbent, self.cfg.thermo, self.cfg.derived
        cp = np.asarray(self.props.cp)
        A = so.total_voidage * (cp[0] * c[0] + cp[1] * c[1] + cp[2] * c[2]) \
            + d.bulk_density * (so.cp_solid + (th.cp_ads_co2 * q[0] + th.cp_ads_h2o * q[1]))
        B = so.total_voidage * host.R_GAS * (c[0] + c[1] + c[2])
        H = d.bulk_density * (th.dH_ads_co2 * q[0] + th.dH_ads_h2o * q[1])
        return A, B, H

    def pack(self, st):
        A, B, H = self._heat(st.c, st.q)
        e = A * (st.T - self.cfg.thermo.T_ref) - B * st.T + H
        return np.concatenate([st.c.ravel(), st.q.ravel(), e.ravel(), st.Tw.ravel()])

    @staticmethod
    def _toth(p, T, qinf, chi, b0, dH, tau0, alpha, T0):
        b = b0 * np.exp(-dH / (host.R_GAS * T)) * p
        tau = tau0 + alpha * (1.0 - T0 / T)
        return qinf * np.exp(chi * (1.0 - T / T0)) * b / (1.0 + b ** tau) ** (1.0 / tau)

    def _loading(self, c, q, T):
        iso = self.cfg.isotherm
        h, co2, wd = iso.h2o, iso.co2, iso.coadsorption.wadst
        RT = host.R_GAS * T
        Tc = T - 273.15
        psat = 611.21 * np.exp((18.678 - Tc / 234.5) * (Tc / (257.14 + Tc)))
        x = np.maximum(c[1] * RT / psat, -0.2)
        over = np.maximum(x - (h.rh_cap - 0.02), 0.0)
        x = np.where(over <= 0.0, x, np.where(over >= 0.04, h.rh_cap, h.rh_cap - 0.02 + over - over ** 2 / 0.08))
        E10 = h.E10_slope * T + h.E10_intercept
        cg = np.exp((h.C - np.exp(h.D * T) - E10) / RT)
        kx = np.exp((h.F + h.G * T - E10) / RT) * x
        qw = h.q_m * cg * kx / ((1.0 - kx) * (1.0 + (cg - 1.0) * kx))
        p = np.maximum(c[0] * RT, 0.0)
        w = np.exp(-wd.A / np.maximum(q[1], 1e-12))
        dry = self._toth(p, T, co2.q_inf0, co2.chi, co2.b0, co2.dH0, co2.tau0, co2.alpha, co2.T0)
        wet = self._toth(p, T, wd.q_inf0_wet, wd.chi_wet, wd.b0_wet, wd.dH_wet, wd.tau0_wet, wd.alpha_wet, co2.T0)
        return ((1.0 - w) * dry + w * wet) * (p / (p + co2.p_regularization)), qw

    def _gas(self, y, T, P):
        mu = np.stack([sum(w * (D * T + E) for w, D, E in t) for t in self.props.mu_terms()])
        kk = np.stack([sum(w * k0 * (T / 300.0) ** n for w, k0, n in t) for t in self.props.k_terms()])
        den = [sum(y[j] * ((1.0 + np.sqrt(mu[i] / mu[j]) * self.props.mass_q[i, j]) ** 2 / self.props.wilke_den[i, j]
                           if i != j else 1.0) for j in range(3)) for i in range(3)]
        den = np.maximum(np.stack(den), 1e-30)
        P = np.maximum(P, 1.0)
        D = [1.43e-7 * T ** 1.75 / ((P / 1e5) * host.fuller_const("CO2", b)) for b in ("AIR", "H2O")]
        Dm = (y[2] + y[1] + 1e-9) / (y[2] / D[0] + y[1] / D[1] + 1e-9 / D[0])
        return (y * mu / den).sum(0), (y * kk / den).sum(0), Dm

    def _stagnant(self, kg):
        tr, so = self.cfg.transport, self.cfg.sorbent
        e = so.bed_voidage
        B, s = tr.zs_shape_factor * ((1.0 - e) / e) ** (10.0 / 9.0), np.sqrt(1.0 - e)
        kap = so.particle_conductivity / kg
        m = 1.0 - B / kap
        kc = (2.0 / m) * ((1.0 - 1.0 / kap) * B / m ** 2 * np.log(kap / B) - 0.5 * (B + 1.0) - (B - 1.0) / m)
        return kg * (1.0 - s + s * kc)

    def _wall_R(self, lam0, Cp, cpm, rho, mu, kg):
        tr, so, g = self.cfg.transport, self.cfg.sorbent, self.g
        dp = so.particle_diameter
        lam = lam0 + Cp * cpm * self.unom * dp / tr.Pe_heat_radial_inf
        Pr = cpm / np.maximum(rho / Cp, 1e-6) * mu / kg
        nu = (1.3 + 5.0 * dp / (2.0 * g.R)) * lam0 / kg
        if self.unom:
            Re = np.maximum(rho * self.unom * dp / mu, 1e-12)
            nu = nu + 1.0 / (1.0 / (0.3 * Pr ** (1.0 / 3.0) * Re ** 0.75) + 1.0 / (0.054 * Pr * Re))
        return dp / (nu * kg) + g.half_dr_outer / lam

    def _end(self, end, t, c, T, P, mu, rho, a, b):
        """Molar inflow per species and enthalpy inflow through a column end."""
        e, g, th = self.cond[end], self.g, self.cfg.thermo
        cp = np.asarray(self.props.cp)[:, None, None]
        yx = None if e.y_ext is None else np.asarray(e.y_ext)[:, None, None]
        Az = g.Az * np.ones_like(T)
        Cc = np.maximum(c.sum(0), 1e-12)
        if e.kind == "closed":
            return np.zeros_like(c), np.zeros_like(T)
        if e.kind == "feed":
            F = self.Fin * yx
            return F, (cp * F).sum(0) * (e.T_ext - th.T_ref)
        if e.kind == "pump":
            dp = np.logaddexp(0.0, P - e.P_target) if e.check_valve else P - e.P_target
            w = 1.0 if e.check_valve else 0.5 * (1.0 + np.tanh(dp / 0.2))
            F = e.speed * dp / (host.R_GAS * T) * Az * (w * c / Cc + (1.0 - w) * yx)
            return -F, -(cp * F).sum(0) * (w * T + (1.0 - w) * e.T_ext - th.T_ref)
        tau = self.cfg.operation.valve_time_constant
        Pr = e.P_target + (self.P0[end] - e.P_target) * np.exp(-t / tau) if tau > 0 else e.P_target
        n_in = e.speed * 0.2 * np.logaddexp(0.0, (Pr - P) / 0.2) / (host.R_GAS * e.T_ext)
        n_out = e.speed * 0.2 * np.logaddexp(0.0, (P - Pr) / 0.2) / (host.R_GAS * T)
        Fi, Fo = n_in * Az * yx, n_out * Az * c / Cc
        return Fi - Fo, (cp * Fi).sum(0) * (e.T_ext - th.T_ref) - (cp * Fo).sum(0) * (T - th.T_ref)

    def __call__(self, t, yv):
        cfg, g = self.cfg, self.g
        so, tr, th, kin = cfg.sorbent, cfg.transport, cfg.thermo, cfg.kinetics
        n, rho_b, eps = g.ncell, cfg.derived.bulk_density, so.bed_voidage
        c = yv[:3 * n].reshape((3,) + g.shape)
        q = yv[3 * n:5 * n].reshape((2,) + g.shape)
        e = yv[5 * n:6 * n].reshape(g.shape)
        Tw = yv[6 * n:].reshape(g.wall_shape)
        A, B, H = self._heat(c, q)
        T = (e - H + A * th.T_ref) / (A - B)
        Ct = c.sum(0)
        P = Ct * host.R_GAS * T
        Tp, Cp = np.clip(T, 150.0, 1500.0), np.maximum(Ct, 1e-9)
        y = c / Cp
        yc = np.clip(y, 0.0, 1.0)
        cp = np.asarray(self.props.cp)
        mu, kg, Dm = self._gas(yc, Tp, P)
        rho, cpm = Cp * np.tensordot(self.props.M, yc, 1), np.tensordot(cp, yc, 1)
        lam0 = self._stagnant(kg)
        qs = self._loading(c, q, Tp)
        rate = [k * np.exp(-E / host.R_GAS * (1.0 / Tp - 1.0 / kin.T_ref)) * (qs[i] - q[i])
                for i, (k, E) in enumerate(((kin.k_ldf_co2, kin.Ea_co2), (kin.k_ldf_h2o, kin.Ea_h2o)))]
        dp = so.particle_diameter
        ka = tr.ergun_A * (1.0 - eps) ** 2 / (eps ** 3 * dp ** 2)
        kb = tr.ergun_B * (1.0 - eps) / (eps ** 3 * dp)

        def velocity(dP, m, r):
            a, b = ka * m, kb * r
            return -2.0 * dP / (a + np.sqrt(a * a + 4.0 * b * np.abs(dP)))

        def enth(F, Tf):
            return np.tensordot(cp, F, 1) * (Tf - th.T_ref)

        def flux(a, b, dist, area, slopes, disp, extra):
            """Species and enthalpy flux from the cells `a` to the cells `b` of a face."""
            mean = lambda x: 0.5 * (a(x) + b(x))                                       # noqa: E731
            u = velocity((b(P) - a(P)) / dist, mean(mu), mean(rho))
            w = 0.5 * (1.0 + np.tanh(u / 1e-4))
            up = lambda x, s: w * (a(x) + 0.5 * a(s)) + (1.0 - w) * (b(x) - 0.5 * b(s))  # noqa: E731
            Fc = u * area * np.stack([up(c[k], slopes[k]) for k in range(3)])
            C = mean(Cp)
            J = -eps * disp(mean(Dm), C) * C / dist * area * np.stack([b(y[k]) - a(y[k]) for k in range(3)])
            lam = mean(lam0) + extra(C * mean(cpm), C)
            return Fc + J, enth(Fc, up(T, slopes[3])) + enth(J, mean(T)) - lam * (b(T) - a(T)) / dist * area

        zero = [np.zeros(g.shape)] * 4
        sl = [np.zeros(g.shape) for _ in range(4)]
        if g.Nz >= 3:
            for s, x in zip(sl, (c[0], c[1], c[2], T)):
                d = np.diff(x, axis=2)
                m, p = d[..., :-1], d[..., 1:]
                s[..., 1:-1] = m * p * (m + p) / (m * m + p * p + 1e-300)

        def disp_z(D, C):
            v = np.abs(self.Nnom / C) / eps
            return tr.er_gamma1 * D + tr.er_gamma2 * dp * v / (1.0 + tr.er_beta * tr.er_gamma1 * D / (dp * v + 1e-30))

        div = np.zeros((3,) + g.shape)
        dE = np.zeros(g.shape)
        F, Hf = flux(lambda x: x[..., :-1], lambda x: x[..., 1:], g.dz, g.Az[:, :, None], sl, disp_z,
                     lambda cc, C: cc * np.abs(self.Nnom / C) * dp / tr.Pe_heat_axial_inf)
        div[..., :-1] += F
        div[..., 1:] -= F
        dE[..., :-1] += Hf
        dE[..., 1:] -= Hf
        for end, k in (("top", 0), ("bottom", -1)):
            F, Hf = self._end(end, t, c[..., k], T[..., k], P[..., k], mu[..., k], rho[..., k], ka, kb)
            div[..., k] -= F
            dE[..., k] -= Hf
        disp_t = lambda D, C: tr.er_gamma1 * D + dp * self.unom / eps / tr.Pe_mass_radial_inf   # noqa: E731
        cond_t = lambda cc, C: cc * self.unom * dp / tr.Pe_heat_radial_inf                      # noqa: E731
        if g.Nr > 1:
            F, Hf = flux(lambda x: x[:-1], lambda x: x[1:], g.drc, g.Ar, zero, disp_t, cond_t)
            div[:, :-1] += F
            div[:, 1:] -= F
            dE[:-1] += Hf
            dE[1:] -= Hf
        if g.Nth > 1:
            F, Hf = flux(lambda x: x, lambda x: np.roll(x, -1, axis=1), g.arc, g.Ath, zero, disp_t, cond_t)
            div += F - np.roll(F, 1, axis=2)
            dE += Hf - np.roll(Hf, 1, axis=1)
        dc = -div / (so.total_voidage * g.V)
        dc[0] -= rho_b / so.total_voidage * rate[0]
        dc[1] -= rho_b / so.total_voidage * rate[1]
        # wall, jacket and ambient
        o = -1
        Tj = float(self.step["jacket"].get("T", cfg.ambient.T))
        Rb = self._wall_R(lam0[o], Cp[o], cpm[o], rho[o], mu[o], kg[o])
        w, jk = cfg.wall, cfg.jacket
        Qj = self.cov * jk.h_jacket * g.A_wall_out * (Tj - Tw)
        Qa = (1.0 - self.cov) * jk.h_ambient * g.A_wall_out * (cfg.ambient.T - Tw)
        Qb = g.A_wall_in * (Tw - T[o]) / Rb
        cond = np.zeros_like(Tw)
        kz = w.conductivity * g.A_wall_axial / g.dz
        cond[:, :-1] += kz * np.diff(Tw, axis=1)
        cond[:, 1:] -= kz * np.diff(Tw, axis=1)
        if g.Nth > 1:
            kt = w.conductivity * g.wall_thickness * g.dz / (g.R_wall_mid * g.dth)
            cond += kt * (np.roll(Tw, -1, 0) - 2.0 * Tw + np.roll(Tw, 1, 0))
        dTw = (Qj + Qa - Qb + cond) / (w.density * w.cp * g.V_wall)
        src = np.zeros(g.shape)
        src[o] = Qb
        de = (-dE + src) / g.V
        return np.concatenate([dc.ravel(), rate[0].ravel(), rate[1].ravel(), de.ravel(), dTw.ravel()])

    def jacobian(self, t, y):
        """Difference quotients in the library's layout J[slot][row][column][cell]: all columns whose
        stencils do not touch perturbed at once."""
        g = self.g
        n, shape = g.ncell, g.shape
        i, j, k = np.meshgrid(*(np.arange(m) for m in shape), indexing="ij")
        # sectors at least three apart around the ring share a group
        groups = np.zeros(g.Nth, dtype=int)
        for a in range(1, g.Nth):
            near = {groups[b] for b in range(a) if min(a - b, g.Nth - a + b) < 3}
            groups[a] = next(x for x in range(g.Nth) if x not in near)
        rho_cp = self.cfg.derived.bulk_density * self.cfg.sorbent.cp_solid
        typ = (1e-3, 1e-2, 1.0, 1e-3, 1e-3, rho_cp, 1.0)
        f0 = self(t, y)
        J = np.zeros((9, 7, 7) + shape)
        slots = [(0, 0, 0), (-1, 0, 0), (1, 0, 0), (-2, 0, 0), (2, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1), (0, 0, 1)]
        for v in range(7):
            base = y[v * n:(v + 1) * n].reshape(shape) if v < 6 else np.broadcast_to(y[6 * n:].reshape(1, g.Nth, g.Nz), shape)
            h = 1.5e-8 * np.maximum(np.abs(base), typ[v])
            h = (base + h) - base
            for ci in range(3):
                for cj in range(groups.max() + 1):
                    for ck in range(5):
                        on = (i % 3 == ci) & (groups[j] == cj) & (k % 5 == ck)
                        if v == 6:
                            on &= i == g.Nr - 1
                        if not on.any():
                            continue
                        yp = y.copy()
                        if v < 6:
                            yp[v * n:(v + 1) * n] += np.where(on, h, 0.0).ravel()
                        else:
                            yp[6 * n:] += np.where(on[-1], h[-1], 0.0).ravel()
                        d = self(t, yp) - f0
                        rows = [d[r * n:(r + 1) * n].reshape(shape) for r in range(6)]
                        wall = np.zeros(shape)
                        wall[-1] = d[6 * n:].reshape(g.wall_shape)
                        for s, (dk, di, dj) in enumerate(slots):
                            if dj and g.Nth == 1:
                                continue
                            ni, nj, nk = i + di, (j + dj) % g.Nth, k + dk
                            ok = (ni >= 0) & (ni < g.Nr) & (nk >= 0) & (nk < g.Nz)
                            a, b = np.where(ok, ni, 0), np.where(ok, nk, 0)
                            ok &= on[a, nj, b]
                            hh = h[a, nj, b]
                            for r, x in enumerate(rows + [wall]):
                                J[s, r, v][ok] = (x / hh)[ok]
        return J.ravel()
