"""The work that the chemistry library does for its users, as timed cases.

Each case is one call (or one forward and backward pass) through the package's public entry
points on inputs of the synthetic distributions that the tests and the benchmark use: CHEM
calls with each solver on subdomains from a few columns to a regional domain's share, the
hour of twelve calls replayed from a graph, sensitivities (DDM-3D) and gradients (discrete
adjoint), the aqueous chemistry of a batch of cloudy cells, and the heterogeneous rates of
a grid.  `listed` gives the cases, `draw` others of the same ranges.
"""
from __future__ import annotations

import json
import math
from pathlib import Path

import numpy as np
import torch

from cmaq_gb300.adjoint import Ros3Window
from cmaq_gb300.aqchem import aqchem, aqchem_kinetics
from cmaq_gb300.chem import ChemSolver
from cmaq_gb300.hetchem import hetchem_rates
from cmaq_gb300.synthetic import (hetchem_tables, make_aerosol_cells, make_cloud_cells, make_cloud_columns, make_grid,
                                  manifest, solver_inputs)

CB6, CRACMM = "cb6r5_ae7_aq", "cracmm2"
FIELDS = ("conc", "ta", "qv", "dens", "pres", "seaice", "ocean_szone", "rj", "khetero")

# most cells of a case of each kind (one pass of the listed cases takes milliseconds to about a second)
MOST = {"chem_ros3_cb6": 126000, "chem_ros3_cracmm2": 10800, "chem_hour": 10500, "chem_ebi_cb6": 27800,
        "chem_ebi_cracmm2": 3000, "chem_gear": 250, "adjoint": 8000, "ddm": 3500, "aqchem": 25000, "kinetics": 4000,
        "hetchem_cb6": 1200000, "hetchem_cracmm2": 300000}
LEAST = {"chem_ros3_cb6": 70, "chem_ros3_cracmm2": 40, "chem_hour": 100, "chem_ebi_cb6": 200, "chem_ebi_cracmm2": 50,
         "chem_gear": 10, "adjoint": 30, "ddm": 30, "aqchem": 50, "kinetics": 20, "hetchem_cb6": 500,
         "hetchem_cracmm2": 500}


def listed():
    return [
        # a rank's few columns of a nested or heavily decomposed domain: launches and the stiffest cell's chain
        {"name": "ros3_columns", "kind": "chem_ros3_cb6", "ncols": 7, "nrows": 5, "nlays": 3, "schedule": "queue",
         "plume": 0.0, "het": True},
        # a GPU's share of a regional domain, 35 layers as CMAQ runs them, with urban plumes
        {"name": "ros3_regional", "kind": "chem_ros3_cb6", "ncols": 60, "nrows": 60, "nlays": 35, "schedule": "queue",
         "plume": 0.1, "het": True},
        # the larger mechanism on a subdomain of odd sizes
        {"name": "ros3_cracmm2", "kind": "chem_ros3_cracmm2", "ncols": 31, "nrows": 27, "nlays": 13,
         "schedule": "queue", "plume": 0.0, "het": True},
        # an hour of twelve 5-minute calls from one captured graph
        {"name": "ros3_hour", "kind": "chem_hour", "ncols": 33, "nrows": 29, "nlays": 11, "schedule": "queue",
         "plume": 0.1, "het": False, "nsteps": 12},
        # CMAQ's default solver on a subdomain
        {"name": "ebi_cb6", "kind": "chem_ebi_cb6", "ncols": 41, "nrows": 40, "nlays": 17, "schedule": "queue",
         "plume": 0.0, "het": True},
        # SMVGEAR, the reference solver for accuracy studies, on a small box of cells
        {"name": "gear_cb6", "kind": "chem_gear", "ncols": 9, "nrows": 7, "nlays": 4, "schedule": "queue",
         "plume": 0.0, "het": False},
        # gradients of a differentiable window of two synchronisation steps: forward and backward
        {"name": "adjoint_cb6", "kind": "adjoint", "cells": 8000, "nsync": 2},
        # a CHEM call that carries four first-order sensitivities
        {"name": "ddm_cb6", "kind": "ddm", "ncols": 21, "nrows": 19, "nlays": 9, "schedule": "queue", "plume": 0.0,
         "het": True, "nparam": 4},
        # the whole aqueous chemistry of a region's cloudy cells, and the kinetics of a few
        {"name": "aqchem_clouds", "kind": "aqchem", "cells": 25000, "ispc8": 0, "mtpyrac": 1},
        {"name": "kinetics_few", "kind": "kinetics", "cells": 333, "ispc8": 1, "mtpyrac": 0},
        # heterogeneous rate constants: a quarter of a continental grid, and a subdomain of the larger mechanism
        {"name": "hetchem_cb6", "kind": "hetchem_cb6", "cells": 1200000},
        {"name": "hetchem_cracmm2", "kind": "hetchem_cracmm2", "cells": 100001},
    ]


def draw(rng):
    kind = rng.choice(sorted(MOST))
    n = int(round(math.exp(rng.uniform(math.log(LEAST[kind]), math.log(MOST[kind])))))
    case = {"kind": kind}
    if kind.startswith("chem") or kind == "ddm":
        nlays = min(n, rng.randint(1, 35))
        ncols = max(1, int(math.sqrt(n / nlays) * math.exp(rng.uniform(-0.5, 0.5))))
        case.update(ncols=ncols, nrows=max(1, n // (nlays * ncols)), nlays=nlays,
                    schedule=rng.choice(["queue", "queue", "static"]) if "ros3" in kind else "queue",
                    plume=rng.choice([0.0, 0.1, 0.3]), het=rng.random() < 0.5)
        if kind == "chem_hour":
            case["nsteps"] = rng.randint(2, 12)
        if kind == "ddm":
            case["nparam"] = rng.randint(1, 6)
    else:
        case["cells"] = n
        if kind == "adjoint":
            case["nsync"] = rng.randint(1, 2)
        if kind in ("aqchem", "kinetics"):
            case.update(ispc8=rng.randint(0, 1), mtpyrac=rng.randint(0, 1))
    return case


def _mech(case):
    return CRACMM if case["kind"].endswith("cracmm2") else CB6


def _cells(case):
    return case["cells"] if "cells" in case else case["ncols"] * case["nrows"] * case["nlays"]


def _grid(case, seed):
    return make_grid(_mech(case), case["ncols"], case["nrows"], case["nlays"], seed=seed,
                     plume_fraction=case["plume"], het=case["het"])


def _solver(case, g, solver):
    return ChemSolver(g.mech, ncols=g.ncols, nrows=g.nrows, nlays=g.nlays, nspcsd=g.nspcsd,
                      cgrid_index=g.cgrid_index, rtol=1.0e-3, atol=1.0e-9, schedule=case.get("schedule", "queue"),
                      solver=solver)


def _up(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind.startswith("chem") or kind == "ddm":
        g = _grid(case, seed)
        solver = "ebi" if "ebi" in kind else "gear" if "gear" in kind else "ros3"
        s["solver"] = _solver(case, g, solver)
        s["in"] = {k: _up(getattr(g, k)) for k in FIELDS}
        s["fresh"] = s["in"]["conc"].clone()
        if kind == "ddm":
            rng = np.random.default_rng(seed + 1)
            npar, n = case["nparam"], g.ncell
            sen = np.zeros((g.nspcsd, npar, n), np.float32)
            for p in range(npar):           # dC/d(scaling of a group of species): their own concentrations
                rows = rng.choice(g.cgrid_index - 1, size=6, replace=False)
                sen[rows, p] = g.conc.reshape(g.nspcsd, n)[rows]
            s["sen_fresh"] = _up(sen.reshape(g.nspcsd, npar, *g.ta.shape))
            s["sen"] = s["sen_fresh"].clone()
            mask = np.zeros((npar, len_rxns(g.mech)), np.uint8)
            mask[npar - 1, rng.integers(0, mask.shape[1], 5)] = 1       # the last parameter: reaction rates
            s["mask"] = _up(mask)
    elif kind == "adjoint":
        g = make_grid(CB6, case["cells"], 1, 1, seed=seed)
        s["solver"] = _solver(case, g, "ros3")
        y0, rki, night = solver_inputs(g, s["solver"])
        rng = np.random.default_rng(seed + 1)
        s["window"] = Ros3Window(s["solver"], rki, night, case["nsync"], 5.0)
        s["y0"] = y0.requires_grad_(True)
        s["log_k"] = _up(rng.normal(0.0, 0.05, rki.shape[0])).requires_grad_(True)
        s["emis"] = _up(rng.uniform(0.0, 1.0e-6, y0.shape)).requires_grad_(True)
        s["cost"] = _up(rng.uniform(0.0, 1.0, y0.shape))     # dL/dy: weights of the observed species
    elif kind == "aqchem":
        p, gas, aer, idx, fac = make_cloud_columns(case["cells"], seed=seed, ispc8=case["ispc8"],
                                                   mtpyrac=case["mtpyrac"])
        s.update(params=_up(p.T), gas_fresh=_up(gas.T), aer_fresh=_up(aer.T), idx=idx, fac=fac)
        s["gas"], s["aer"] = s["gas_fresh"].clone(), s["aer_fresh"].clone()
    elif kind == "kinetics":
        p, v = make_cloud_cells(case["cells"], seed=seed, ispc8=case["ispc8"], mtpyrac=case["mtpyrac"])
        s.update(params=_up(p.T), var=_up(v.T))
    else:
        s["in"] = tuple(_up(x) for x in make_aerosol_cells(case["cells"], seed=seed, mech=_mech(case)))
        s["labels"] = hetchem_tables(_mech(case))["hetero"]
    return s


def len_rxns(mech):
    return int(manifest(mech)["nrxns"])


def _totals(st):
    return {k: int(st[k]) for k in ("accepted_steps", "rejected_steps", "failed_cells", "sunlit_cells") if k in st}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind.startswith("chem"):
        f = s["in"]
        f["conc"].copy_(s["fresh"])          # the transported concentrations of a new synchronisation step
        args = [f[k] for k in FIELDS]
        st = s["solver"].steps(case["nsteps"], *args) if kind == "chem_hour" else s["solver"].step(*args)
        return {"conc": f["conc"], "totals": _totals(st)}
    if kind == "ddm":
        f = s["in"]
        f["conc"].copy_(s["fresh"])
        s["sen"].copy_(s["sen_fresh"])
        st = s["solver"].step_ddm(s["sen"], *[f[k] for k in FIELDS], rate_mask=s["mask"])
        return {"conc": f["conc"], "sen": s["sen"], "totals": _totals(st)}
    if kind == "adjoint":
        y = s["window"](s["y0"], s["log_k"], s["emis"])
        gy, gk, ge = torch.autograd.grad(y, (s["y0"], s["log_k"], s["emis"]), s["cost"])
        return {"y": y.detach(), "dy0": gy, "dlog_k": gk, "demis": ge}
    if kind == "aqchem":
        s["gas"].copy_(s["gas_fresh"])
        s["aer"].copy_(s["aer_fresh"])
        gwd, awd, out, stats = aqchem(s["params"], s["gas"], s["aer"], s["idx"], s["fac"])
        return {"gas": s["gas"], "aer": s["aer"], "gas_wdep": gwd, "aer_wdep": awd, "out": out, "stats": stats}
    if kind == "kinetics":
        var, stats = aqchem_kinetics(s["params"], s["var"])
        return {"var": var, "stats": stats}
    kh = hetchem_rates(*s["in"], mechanism=_mech(case))
    return {label: kh[:, j] for j, label in enumerate(s["labels"])}


# FP64 operations (FMA = 2) of one pass: attempts per cell and call of these inputs (the counts that the
# kernels report, day and night cells together) times the operations of an attempt or iteration
_ATTEMPT = {CB6: 36.9e3, CRACMM: 80.0e3}
_ATTEMPTS = {"chem_ros3_cb6": 40.5, "chem_ros3_cracmm2": 76.9, "chem_hour": 8.2, "ddm": 40.0}


def work(case):
    kind, n = case["kind"], _cells(case)
    if kind.startswith("hetchem"):
        rows, het = (84, 17) if kind == "hetchem_cb6" else (90, 9)
        return {"bytes": n * (4.0 * (rows + 4) + 8.0 * het), "flops": n * 2.0e3}
    if kind == "aqchem":
        return {"bytes": n * 8.0 * (15 + 2 * 2 * (29 + 93) + 10 + 5), "flops": n * 0.82e6}
    if kind == "kinetics":
        return {"bytes": n * 8.0 * (15 + 2 * 161 + 5), "flops": n * 0.82e6}
    man = manifest(_mech(case))
    if kind == "adjoint":
        ns, nr = man["nspec"], man["nrxns"]
        return {"bytes": n * 8.0 * (6 * ns + nr) + 16.0 * nr, "flops": n * case["nsync"] * 2.6 * 25 * _ATTEMPT[CB6]}
    per_cell = 4.0 * (2 * man["nspec"] + 4 + len(man["photab"])) + 8.0 * man["nhetero"]
    calls = case.get("nsteps", 1)
    if "ebi" in kind:
        flops = 122 * (1.4e4 if kind.endswith("cracmm2") else 7.0e3)
    elif "gear" in kind:
        flops = 300 * 1.5e4
    else:
        flops = calls * _ATTEMPTS[kind] * _ATTEMPT[_mech(case)]
    if kind == "ddm":
        per_cell += 8.0 * case["nparam"] * man["nspec"]
        flops += 2.0e4 + case["nparam"] * 1.0e4
    return {"bytes": n * per_cell, "flops": n * flops}


def exact(case, seed):
    """HETCHEM_RATES in 64 bits.  The other entry points integrate stiff systems with their own
    step control to a set tolerance: what they return is the numerical solution of their steps,
    which has no value apart from taking them."""
    if not case["kind"].startswith("hetchem"):
        return None
    k = _hetchem64(_mech(case), *make_aerosol_cells(case["cells"], seed=seed, mech=_mech(case)))
    # the split of the IEPOX uptake in clean air hangs on q / TANH( q ) > 1 for q near 1e-8: no value in more digits
    split = ("HETERO_IEPOXOS", "HETERO_TETROL", "HETERO_ISO3NOSJ", "HETERO_ISO3OSJ")
    labels = hetchem_tables(_mech(case))["hetero"]
    return {label: None if label in split else k[:, j] for j, label in enumerate(labels)}


def _hetchem64(mech, ae, ta, pres, qv, dens):
    """KHETERO from the formulas of HETCHEM_RATES (AEROSOL_CHEMISTRY.F), all in 64 bits."""
    t = json.loads((Path(__file__).resolve().parents[1] / "cmaq_gb300" / "mechs" / mech / "hetchem.json").read_text())
    sp, ix = t["species"], t["idx"]
    ae, ta, pres, qv, dens = (np.asarray(x, np.float64) for x in (ae, ta, pres, qv, dens))
    n = ta.size
    f4 = lambda x: float(np.float32(x))          # the reference's REAL(4) parameters
    pi4, dpi, conmin, rgas, mwair, mwwat = f4(3.14159265), math.pi, 1.0e-23, f4(8.31451), f4(28.9628), f4(18.0153)
    f6pi = 6.0 / pi4
    c = np.zeros((len(sp), 3, n))
    for i, s in enumerate(sp):
        for m in range(3):
            if s["row"][m] >= 0:
                c[i, m] = np.maximum(ae[s["row"][m]], s["min_conc"][m])
    mw = np.array([f4(s["molwt"]) for s in sp])
    wet2, wet3, de = np.zeros((3, n)), np.zeros((3, n)), np.zeros((3, n))
    for m in range(3):
        dry = sum(c[i, m] / s["density"] for i, s in enumerate(sp) if not s["no_m2wet"] and not s["tracer"])
        wet = sum(c[i, m] / s["density"] for i, s in enumerate(sp) if not s["tracer"] and s["row"][m] >= 0)
        dry, wet = np.maximum(dry * 1.0e-9 * f6pi, conmin), np.maximum(wet * 1.0e-9 * f6pi, conmin)
        m0 = np.maximum(ae[t["num_rows"][m]], conmin)
        m2 = np.maximum(ae[t["srf_rows"][m]] / pi4, conmin) * (wet / dry) ** (2.0 / 3.0)
        x = np.log(m0) / 3.0 + 2.0 * np.log(wet) / 3.0
        l2 = np.clip(x - np.log(m2), math.log(f4(1.05)) ** 2, math.log(f4(2.5001)) ** 2)
        m0 = np.maximum(m0, wet / (1.0e-12 * np.exp(4.5 * l2)))
        wet2[m], wet3[m] = np.exp(x - l2), wet
        de[m] = np.cbrt(wet / (m0 * np.exp(4.5 * l2))) * np.exp(1.5 * l2)
    eps = mwwat / mwair
    rh = np.clip(pres * qv / (eps + qv) / 610.94 * np.exp(17.625 * (273.15 - ta) / (ta - 273.15 + 243.04)), 0.005, 0.99)
    coeff = np.sqrt(8.0 * 1.0e3 * rgas / pi4 * ta)
    diff = (ta / 273.15) ** 1.75 * (101325.0 / pres)
    ppm, rfac = 1.0e-3 * mwair / dens, 60.0 * 7.24382926227485e10 * pres / ta
    speed = lambda w: np.sqrt(8.0e3 * rgas / (w * dpi)) * np.sqrt(ta)
    cbar, inv_d = coeff * 9.62161363758323e-2, 1.0 / (0.0855e-4 * diff)
    fine = lambda name: c[ix[name], 0] + c[ix[name], 1]
    no3, so4, nh4 = (fine(k) / mw[ix[k]] for k in ("ANO3", "ASO4", "ANH4"))
    with np.errstate(all="ignore"):
        ani = no3 + so4
        logit = lambda v: 1.0 / (1.0 + np.exp(-v))
        x3 = no3 / ani
        x2 = np.clip(np.minimum(1.0 - x3, nh4 / ani - 1.0), 0.0, None)
        x1 = 1.0 - x2 - x3
        gam3 = np.minimum(logit(-8.10774 + 4.902 * rh), 0.0154)
        gamd = np.minimum(logit(-6.13376 + 3.592 * rh - 0.19688 * np.maximum(0.0, ta - 293.0)), 0.0124)
        lam2 = -3.64849 + 9.553 * np.minimum(0.0, rh - 0.46)
        lam1 = lam2 + 0.97579 - 0.20427 * np.maximum(0.0, ta - 291.0)
        aqueous = x1 * np.minimum(logit(lam1), 0.08585) + x2 * np.minimum(logit(lam2), 0.053) + x3 * gam3
        dry = (x1 + x2) * gamd + x3 * np.minimum(gamd, gam3)
        x, y = nh4 / np.maximum(nh4, 2.0 * so4 + no3), so4 / ani
        crh = (3143.44 + 63.07 * x + 0.114 * x * x + 87.97 * y - 125.73 * x * y + 0.586 * x * x * y + 0.95 * y * y
               - 1.384 * x * y * y - 79692.5 / (25.0 + (x - 0.7) * (y - 0.5)))
        crystal = (rh <= 0.01) | ((rh <= 0.351) & (x >= 0.5) & (y >= 0.22) & (rh <= crh))
        eirh = 1.61299 + ta * (4.4117437e-5 * ta - 1.4293888e-2)
        a, b, d, e = 373.16 / ta, ta / 373.16, 273.16 / ta, ta / 273.16
        lw = (-7.90298 * (a - 1.0) + 5.02808 * np.log10(a) - 1.3816e-7 * (10.0 ** (11.344 * (1.0 - b)) - 1.0)
              + 8.1328e-3 * (10.0 ** (-3.49149 * (a - 1.0)) - 1.0) + 3.0057149)
        li = -9.09718 * (d - 1.0) - 3.56654 * np.log10(d) + 0.876793 * (1.0 - e) + 0.78583503
        ice = (ta < 273.16) & ((rh > eirh + 0.005) | ((rh >= eirh - 0.005) & (rh > 10.0 ** (li - lw))))
        gfine = np.where(ice, 0.02, np.where(crystal, dry, aqueous))
        vol = 1.0e-9 * f6pi / wet3[2]
        h2om, clm, no3m = (c[ix[k], 2] * vol / mw[ix[k]] for k in ("AH2O", "ACL", "ANO3"))
        k2f = -1.15e6 * np.expm1(-0.13 * h2om)
        gcoarse = 3.2e-8 * k2f * (1.0 - 1.0 / (0.06 * (h2om / no3m) + 1.0 + 29.0 * (clm / no3m)))
        uptake = lambda m, g, v: g * wet2[m] / (4.0 + 0.5 * de[m] * g * v * inv_d) * v * dpi
        kn = [uptake(m, gfine if m < 2 else gcoarse, cbar) for m in range(3)]
        r_h2ocl = mw[ix["AH2O"]] / mw[ix["ACL"]]

        def clyield(w, cl):
            ok = (w > 0.5) & (cl > 1.0e-4) & (r_h2ocl * cl > 1.0e-4 * w)
            return np.where(ok, 1.0 / (1.0 + w / cl / r_h2ocl / 483.0), 0.0)

        yij, yk = clyield(fine("AH2O"), fine("ACL")), clyield(c[ix["AH2O"], 2], c[ix["ACL"], 2])
        clppm = [ppm * c[ix["ACL"], m] / mw[ix["ACL"]] for m in range(3)]
        # IEPOX uptake
        acid = np.maximum(c[ix["AH3OP"], 1] / mw[ix["AH3OP"]] * 1.0e-6, 0.0)
        charge = -sum(s["charge"] * c[i, 1] / mw[i] for i, s in enumerate(sp) if not s["tracer"] and s["row"][1] >= 0)
        acids = (acid, np.maximum(charge * 1.0e-6 - acid, 0.0))
        ivol = 1.0e6 / sum(c[i, 1] / s["density"] for i, s in enumerate(sp) if not s["tracer"] and s["row"][1] >= 0)
        ktet, kos = np.zeros(n), np.zeros(n)
        for p in t["nuc_pairs"]:
            nuc = c[p["nuc_spc"], 1] / mw[p["nuc_spc"]] * 1.0e-6
            if p["idx_remove"] >= 1:
                nuc = np.maximum(nuc - acids[p["idx_remove"] - 1], 0.0)
            k = p["kchem"] * nuc * acids[p["idx_acid"] - 1] * ivol * ivol
            ktet, kos = (ktet, kos + k) if p["os"] else (ktet + k, kos)
        kp = ktet + kos
        rad_i, rad = 0.5 * de[0], 0.5 * de[1]
        q = rad * np.sqrt(kp / 1.0e-9)
        qm1 = np.where(q < 0.1, q * q / 3.0 * (1.0 - q * q / 15.0 * (1.0 - 2.0 * q * q / 21.0)), q / np.tanh(q) - 1.0)
        heff = t["henry_iepox"][0] * np.exp(t["henry_iepox"][1] * (298.0 - ta) / (298.0 * ta))
        nu = speed(t["gas_molwt"]["IEPOX"])
        up = q / np.tanh(q) > 1.0
        gi = np.where(up, 1.0 / (50.0 + nu * rad / (4.0 * heff * 0.08206 * ta * 1.0e-9 * qm1)), 0.0)
        ftet, fos = np.where(up, ktet / kp, 0.0), np.where(up, kos / kp, 0.0)
        on = gi > 1.0e-72
        kiepox = np.where(on, wet2[1] * dpi / (rad * inv_d + 4.0 / (nu * gi)), 0.0)
        so4ppm = np.where(on, ppm * c[ix["ASO4"], 1] / mw[ix["ASO4"]], 0.0)
        toa = sum(c[i, 0] + c[i, 1] for i, s in enumerate(sp) if s["om"] and not s["tracer"])
        part = np.where(toa >= 1.0e-4, 0.34 / (1.0 + 0.73 / toa) + 0.66 / (1.0 + 1000.0 / toa), 0.0)
        ntr2 = part * 2.7778e-3 * np.clip(5.0 * rh - 1.0, 0.0, 1.0)
        h2o_time = 4.0 / 0.024 / (coeff * 1.012739360000e-1)
        inv_dc = 1.0 / (0.1014e-4 * diff)

        def pncom(m):
            poc, nc = c[ix["APOC"], m], c[ix["APNCOM"], m]
            r = (poc + nc) / poc
            v = np.where(r >= 11.0 / 3.0, 15.0 / 16.0 * 2.5e-12,
                         15.0 * 2.5e-12 / (16.0 + (11.0 / 3.0 - r) / (r - 7.0 / 6.0)))
            return rfac * np.where((poc <= 1.0e-30) | (r <= 7.0 / 6.0), 0.0, v)

        gas = lambda key, g, m: uptake(m, g, speed(t["gas_molwt"][key]))
        mgly = f4(0.09) * 2.9e-3
        os = np.where(so4ppm > 0.0, 6.0e10 * fos / so4ppm, 0.0)
        rate = {
            "N2O5IJ": 60.0 * (kn[0] + kn[1]), "N2O5K": 60.0 * kn[2], "H2NO3PAIJ": 6.0e10 * (1.0 - yij),
            "H2NO3PBIJ": np.where(yij > 0.0, 6.0e10 * yij / (clppm[0] + clppm[1]), 0.0),
            "H2NO3PAK": 6.0e10 * (1.0 - yk), "H2NO3PBK": np.where(yk > 0.0, 6.0e10 * yk / clppm[2], 0.0),
            "PNCOMLI": pncom(0), "PNCOMLJ": pncom(1), "NO2": 60.0e-4 * (wet2[0] + wet2[1]) * dpi,
            "IEPOX": 60.0 * kiepox, "TETROL": 6.0e10 * ftet, "ISO3NOSJ": 6.0e10 * ftet, "IEPOXOS": os, "ISO3OSJ": os,
            "NO3": 60.0 * (gas("NO3", 1.0e-3, 0) + gas("NO3", 1.0e-3, 1)), "GLY": 60.0 * gas("GLY", 2.9e-3, 1),
            "MGLY": 60.0 * gas("MGLY", mgly, 1), "HO2": 60.0 * gas("HO2", 0.2, 1), "NTR2": ntr2,
            "CLNO3_WAI": 60.0 * wet2[0] * dpi / (rad_i * inv_dc + h2o_time),
            "CLNO3_WAJ": 60.0 * wet2[1] * dpi / (rad * inv_dc + h2o_time),
        }
    return np.stack([rate[h.removeprefix("HETERO_")] for h in t["hetero"]], axis=1)
