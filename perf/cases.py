"""The work a user of this framework has it do, as timed cases.

Every case goes through the public Python entry points (``revsim.water``, ``revsim.sw``,
``revsim.gas`` and ``revsim.Engine``) with host arrays in and host arrays out, as the
reference's own driver scripts call them.  The kinds:

* ``forces``    one evaluation of a configuration: forces, energy and dE/dtheta;
* ``train``     one update of train(): forward_sim, then reverse_sim over the same window
                (optionally several boxes in one engine, any pair form, the learned term);
* ``reweight``  reweighting_sim, the ensemble-reweighting gradient estimator;
* ``equil``     a barostatted equilibration run (forward only);
* ``diamond``   one update of the Stillinger-Weber diamond training (stress loss);
* ``gas``       one update of the gas-diffusion training (diffusion, RDF and enthalpy losses).

Windows are short (train() truncates its reverse windows too) so that outputs stay
comparable: over a thousand steps two roundings of the same trajectory part ways.  Results
of a mixed-precision engine are FP32 results and are returned as such.
"""

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "rev-sim_b200"))

from revsim import Engine, SwEngine, constants as C, diamond as D, gas, loss, mlp, sw, systems, water  # noqa: E402

MLP_SEED = 3


# --------------------------------------------------------------------------- cases
def listed():
    """The listed cases; each comment says what it stands for in real use."""
    return [
        # the smallest call: score one small configuration (line searches, checks, examples)
        dict(name="forces_150_fp64", kind="forces", n_mol=150, box=2.6, inter="lj", precision="fp64"),
        # the reference's own training update: 895 waters (tip3p.pdb's box), RDF + enthalpy loss
        # on the experimental grid, plain FP64
        dict(name="train_895_lj_both_fp64", kind="train", n_mol=895, box=3.0, reps=1, spread=False,
             inter="lj", precision="fp64", loss="both", mlp=False, exact=False, gamma=1.0, steps=120,
             every=60, trunc=60),
        # the same box with the double-exponential form in mixed precision, RDF loss alone
        dict(name="train_895_dexp_rdf_mixed", kind="train", n_mol=895, box=3.0, reps=1, spread=False,
             inter="dexp", precision="mixed", loss="rdf", mlp=False, exact=False, gamma=1.0, steps=60,
             every=60, trunc=60),
        # the headline benchmark's box and settings, a short window of it
        dict(name="headline_3000_lj_mixed", kind="train", n_mol=3000, box=4.5, reps=1, spread=False,
             inter="lj", precision="mixed", loss="l2", mlp=False, exact=True, gamma=0.0, steps=60,
             every=60, trunc=60),
        # the same system in plain FP64 (the comparison arm of every result), an odd molecule count
        dict(name="train_2001_buck_fp64", kind="train", n_mol=2001, box=3.94, reps=1, spread=False,
             inter="buck", precision="fp64", loss="l2", mlp=False, exact=False, gamma=1.0, steps=60,
             every=60, trunc=60),
        # the batched target configuration: sixteen 895-water boxes in one engine
        dict(name="batch_16x895_lj_mixed", kind="train", n_mol=895, box=3.0, reps=16, spread=False,
             inter="lj", precision="mixed", loss="l2", mlp=False, exact=True, gamma=0.0, steps=40,
             every=40, trunc=40),
        # the replica benchmark: 64 ragged boxes of 300 to 3,000 waters at their own temperatures
        dict(name="batch_64_ragged_lj_mixed", kind="train", n_mol=3000, box=0.0, reps=64, spread=True,
             inter="lj", precision="mixed", loss="l2", mlp=False, exact=False, gamma=1.0, steps=24,
             every=24, trunc=24),
        # training the learned pair correction on the 895-water box
        dict(name="train_895_mlp_mixed", kind="train", n_mol=895, box=3.0, reps=1, spread=False,
             inter="lj", precision="mixed", loss="l2", mlp=True, exact=True, gamma=0.0, steps=60,
             every=60, trunc=60),
        # the reweighting estimator, loss points close together
        dict(name="reweight_895_lj_fp64", kind="reweight", n_mol=895, box=3.0, inter="lj",
             precision="fp64", loss="both", gamma=1.0, steps=100, every=20),
        # barostatted equilibration of the headline box
        dict(name="equil_3000_lj_mixed", kind="equil", n_mol=3000, box=4.5, inter="lj",
             precision="mixed", gamma=5.0, steps=60),
        # the diamond benchmark: 16 x 8,000 atoms with the learned radial term
        dict(name="diamond_16x8000_mlp_mixed", kind="diamond", cells=10, reps=16, mlp=True,
             precision="mixed", gamma=4.0, steps=24, every=12),
        # the gas-diffusion training update: 885 waters and 10 O2, all three losses, plain FP64
        dict(name="gas_885_10_lj_fp64", kind="gas", n_water=885, n_gas=10, box=3.0, inter="lj",
             precision="fp64", loss="diff_rdf_ev", gamma=1.0, steps=120, every=60, trunc=60),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box_for(rng, n_mol, least=2.5):
    """A box at liquid density within a few per cent, at least `least` (the list cutoff needs
    2.4 nm)."""
    return round(max(least, (n_mol / rng.uniform(31.5, 34.0)) ** (1.0 / 3.0)), 3)


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    kind = rng.choice(["forces", "train", "train", "train", "batch", "mlp", "reweight", "equil",
                       "diamond", "gas"])
    inter = rng.choice(["lj", "lj", "dexp", "buck", "ljsc", "buff"])
    precision = rng.choice(["fp64", "mixed"])
    n = _log_int(rng, 150, 3000)
    if kind == "forces":
        return dict(kind="forces", n_mol=n, box=_box_for(rng, n), inter=inter, precision=precision)
    if kind == "reweight":
        every = rng.randint(10, 30)
        n = _log_int(rng, 300, 3000)
        return dict(kind="reweight", n_mol=n, box=_box_for(rng, n), inter=inter, precision=precision,
                    loss=rng.choice(["rdf", "both"]), gamma=1.0, steps=every * rng.randint(2, 5),
                    every=every)
    if kind == "equil":
        n = _log_int(rng, 600, 3000)
        return dict(kind="equil", n_mol=n, box=_box_for(rng, n, 2.6), inter=inter, precision=precision,
                    gamma=rng.choice([1.0, 5.0]), steps=rng.randint(35, 75))
    if kind == "diamond":
        every = rng.randint(6, 12)
        cells = rng.randint(4, 10)
        reps = rng.randint(1, 16)
        return dict(kind="diamond", cells=cells, reps=reps, mlp=rng.random() < 0.5, precision=precision,
                    gamma=4.0, steps=2 * every, every=every)
    if kind == "gas":
        every = rng.randint(20, 60 if precision == "fp64" else 30)
        nw = _log_int(rng, 500, 1500)
        ng = rng.randint(1, 20)
        return dict(kind="gas", n_water=nw, n_gas=ng, box=_box_for(rng, nw + ng), inter=inter,
                    precision=precision, loss=rng.choice(["diff", "diff_ev", "diff_rdf_ev"]), gamma=1.0,
                    steps=2 * every, every=every, trunc=rng.randint(10, every))
    every = rng.randint(20, 60)
    case = dict(kind="train", n_mol=n, box=_box_for(rng, n), reps=1, spread=False, inter=inter,
                precision=precision, loss=rng.choice(["l2", "rdf", "both"]), mlp=False, exact=False,
                gamma=1.0, steps=every * rng.randint(1, 2), every=every, trunc=every)
    if rng.random() < 0.4:
        case.update(gamma=0.0, exact=True)
    if case["precision"] == "mixed":
        case["steps"] = every
    if kind == "mlp":
        case.update(inter="lj", mlp=True, loss="l2", n_mol=_log_int(rng, 300, 1500))
        case["box"] = _box_for(rng, case["n_mol"])
    if kind == "batch":
        reps = rng.randint(2, 16)
        m = _log_int(rng, 300, 1500)
        s = rng.randint(14, 24)
        case.update(reps=reps, n_mol=m, loss="l2", spread=rng.random() < 0.5, steps=s, every=s, trunc=s)
        case["box"] = _box_for(rng, m)
    return case


# ------------------------------------------------------------------- what a case needs
def _sizes(case, seed):
    """(molecules, box side, temperature) per replica of a water case."""
    if case.get("spread"):
        rng = np.random.default_rng(2)
        n = np.exp(rng.uniform(np.log(300), np.log(case["n_mol"]), case["reps"])).astype(int)
        temps = rng.uniform(280.0, 320.0, case["reps"])
        box = np.maximum(2.45, (n / 33.1) ** (1.0 / 3.0))
        return list(n), list(box), list(temps)
    r = case.get("reps", 1)
    return [case["n_mol"]] * r, [case["box"]] * r, [C.TEMP] * r


def _pairs(n_atoms, box):
    """Unordered atom pairs within the 1.0 nm cutoff at uniform density."""
    return 0.5 * n_atoms * n_atoms * (4.0 / 3.0) * math.pi / box ** 3


def work(case):
    """Bytes (inputs once, outputs once) and operations (pairs within the cutoff, 55 per pair
    and forward step, 170 per pair and reverse step; the diamond terms by active neighbour)."""
    k = case["kind"]
    if k == "diamond":
        n = 8 * case["cells"] ** 3 * case["reps"]
        per_fwd = 18 * 9.7 * 8.7 + 40 * 9.7
        per_rev = 97 * 9.7 * 8.7 + 440 * 9.7
        return {"bytes": 8.0 * 3 * n * 6, "flops": n * case["steps"] * (per_fwd + per_rev)}
    if k == "gas":
        n = 3 * case["n_water"] + 2 * case["n_gas"]
        p = _pairs(n, case["box"])
        rev = 2 * min(case["trunc"], case["every"])
        return {"bytes": 8.0 * 3 * n * 6, "flops": p * (55.0 * case["steps"] + 170.0 * rev)}
    ns, boxes, _ = _sizes(case, 0)
    n = 3 * int(sum(ns))
    p = sum(_pairs(3 * m, b) for m, b in zip(ns, boxes))
    if k == "forces":
        return {"bytes": 8.0 * 3 * n * 3, "flops": 85.0 * p}
    if k == "train":
        rev = case["steps"] // case["every"] * case["trunc"]
        return {"bytes": 8.0 * 3 * n * 6, "flops": p * (55.0 * case["steps"] + 170.0 * rev)}
    if k == "reweight":
        return {"bytes": 8.0 * 3 * n * 4, "flops": p * (55.0 * case["steps"] + 30.0 * (case["steps"] // case["every"]))}
    return {"bytes": 8.0 * 3 * n * 4, "flops": p * 55.0 * case["steps"]}


# --------------------------------------------------------------------------- inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _faces_in_gaps(x, box):
    """Translate a periodic configuration so that the box faces lie in the widest gap of the
    coordinates along each axis: no atom starts on a face, where one rounding would move it to
    the other side of the box."""
    out = x.copy()
    for u in range(3):
        c = np.sort(x[:, u])
        gaps = np.diff(np.append(c, c[0] + box))
        k = int(np.argmax(gaps))
        out[:, u] -= c[k] + 0.5 * gaps[k]
    return out - np.floor(out / box) * box


def _relaxed(ns, boxes, temps, seeds, gas_mol=None):
    """Liquid-like positions of several boxes: seeded lattices relaxed together by 0.15 ps of
    strongly damped Langevin dynamics in plain torch (FP32, short cutoff), so that the timed
    dynamics start near equilibrium and not from the lattice's random orientations."""
    models, xs, tabs, o = [], [], [], 0
    theta = C.default_params("lj") if gas_mol is None else C.gas_default_params("lj")
    for n, b, seed in zip(ns, boxes, seeds):
        x = systems.water_coords(n, b, seed=seed).reshape(n, 3, 3)
        if gas_mol is not None and len(gas_mol):
            d = x[gas_mol, 1] - x[gas_mol, 0]
            d -= b * np.round(d / b)
            x[gas_mol, 1] = x[gas_mol, 0] + d / np.linalg.norm(d, axis=1, keepdims=True) * C.GAS_R0_BOND
            x[gas_mol, 2] = x[gas_mol, 1]
        M = _Model("lj", theta, n, b, rc=0.55, dtype=torch.float32, gas_mol=gas_mol)
        q = torch.tensor(x, dtype=torch.float32, device=M.dev)
        idx, val = M.table(q, skin=0.2)
        models.append(M)
        xs.append(q)
        tabs.append((idx + o, val))
        o += n
    dev, K = models[0].dev, max(t[0].shape[1] for t in tabs)
    pad = torch.nn.functional.pad
    idx = torch.cat([pad(t[0], (0, K - t[0].shape[1])) for t in tabs])
    val = torch.cat([pad(t[1], (0, K - t[1].shape[1])) for t in tabs])
    M = models[0]
    M.q, M.on, M.is_gas, M.mass = (torch.cat([getattr(m, k) for m in models]) for k in ("q", "on", "is_gas", "mass"))
    per_mol = lambda v: torch.repeat_interleave(torch.tensor(np.asarray(v), dtype=torch.float32, device=dev),  # noqa: E731
                                                torch.tensor(np.asarray(ns), device=dev))
    L, kT = per_mol(boxes), C.KB * per_mol(temps)
    q, mass = torch.cat(xs), M.mass[:, :, None]
    g = torch.Generator(device=dev)
    g.manual_seed(int(seeds[0]) % (1 << 31))
    sd = torch.sqrt(kT[:, None, None] / mass)
    v = torch.randn(q.shape, generator=g, device=dev) * sd
    dt, gam = 0.001, 30.0
    c = math.exp(-gam * dt)
    s = math.sqrt(1 - c * c)
    for _ in range(150):
        f = M.forces_fast(q, (idx, val), L)
        v = (v + f / mass * dt) * c + torch.randn(q.shape, generator=g, device=dev) * sd * s
        step = (v * dt).clamp(-0.004, 0.004)
        q = q + step
        v = step / dt
        if gas_mol is not None and len(gas_mol):
            q[M.gas_idx, 2] = q[M.gas_idx, 1]
    y, out, o = q.double().cpu().numpy(), [], 0
    for n, b in zip(ns, boxes):
        w = y[o:o + n].reshape(-1, 3)
        out.append(_faces_in_gaps(w - np.floor(w / b) * b, b))
        o += n
    return out


def _water_inputs(case, seed):
    ns, boxes, temps = _sizes(case, seed)
    ns = [int(n) for n in ns]
    xs = _relaxed(ns, boxes, temps, [1000 * seed + r for r in range(len(ns))])
    vs = [systems.mb_velocities(n, temp=t, seed=1000 * seed + 500 + r) for r, (n, t) in enumerate(zip(ns, temps))]
    return np.concatenate(xs), np.concatenate(vs), ns, boxes, temps


def _targets(case, seed):
    """RDF terms: the experimental-grid L1 terms or the 200-bin O-O L2 term, against smooth
    synthetic curves (the experimental file is not part of this repository)."""
    rng = np.random.default_rng(7000 + seed)
    if case["loss"] in ("rdf", "both", "diff_rdf_ev"):
        k = np.arange(281)
        shape = 1.0 + 0.3 * np.sin(0.07 * k + rng.uniform(0, 1)) * np.exp(-k / 150.0)
        return loss.reference_rdf_terms(shape[:248], shape)
    r = (np.arange(200) + 1) * 0.005
    return [loss.oo_l2_term(1.0 / (1.0 + np.exp(-(r - 0.26) / 0.008)) * (1 + 0.2 * np.cos(20 * r + rng.uniform(0, 1))))]


def _theta(case, seed):
    p = np.array(C.default_params(case["inter"]))
    p = p * (1.0 + 0.002 * np.random.default_rng(8000 + seed).uniform(-1, 1, len(p)))
    if case.get("mlp"):
        p = np.concatenate([p, mlp.init_params(MLP_SEED)])
    return p


def prepare(case, seed):
    """What a program has in hand before the call: start state, parameters, per-step noise
    seeds, loss targets and the engine."""
    k = case["kind"]
    if k == "diamond":
        R, n = case["reps"], 8 * case["cells"] ** 3
        xs, vs = [], []
        for r in range(R):
            x, box = D.diamond_coords(case["cells"], noise=0.004, seed=1000 * seed + r)
            xs.append(_faces_in_gaps(x, box))
            vs.append(D.mb_velocities(n, seed=1000 * seed + 500 + r))
        eng = SwEngine([n] * R, [box] * R, precision=case["precision"], mlp=case["mlp"])
        rng = np.random.default_rng(8000 + seed)
        return dict(case=case, eng=eng, x=np.concatenate(xs), v=np.concatenate(vs), box=box,
                    p=D.default_params() * (1.0 + 0.002 * rng.uniform(-1, 1, 7)),
                    pm=D.init_mlp_params(MLP_SEED) if case["mlp"] else None,
                    target=np.diag([-400.0, -380.0, -420.0]) + rng.uniform(-20, 20, (3, 3)),
                    seeds=systems.noise_seeds(case["steps"], seed))
    if k == "gas":
        nw, ng = case["n_water"], case["n_gas"]
        n = nw + ng
        g = np.arange(nw, n)
        order = np.random.default_rng(6000 + seed).permutation(n)   # which molecules become gas
        gm = np.sort(order[:ng])
        x = _relaxed([n], [case["box"]], [C.TEMP], [1000 * seed], gas_mol=gm)[0].reshape(n, 3, 3)
        keep = np.setdiff1d(np.arange(n), gm)
        x = np.concatenate([x[keep].reshape(-1, 3), x[gm, :2].reshape(-1, 3)])
        p = np.array(C.gas_default_params(case["inter"]))
        p = p * (1.0 + 0.002 * np.random.default_rng(8000 + seed).uniform(-1, 1, len(p)))
        eng = gas.GasEngine(nw, ng, case["box"], case["inter"], precision=case["precision"])
        return dict(case=case, eng=eng, x=x, v=systems.gas_water_velocities(nw, ng, seed=1000 * seed + 1), p=p,
                    terms=_targets(case, seed) if "rdf" in case["loss"] else None, gas=g,
                    seeds=systems.noise_seeds(case["steps"], seed))
    x, v, ns, boxes, temps = _water_inputs(case, seed)
    one = len(ns) == 1
    eng = Engine(ns[0] if one else ns, boxes[0] if one else boxes, temp=temps[0] if one else temps,
                 inter_type=case["inter"], precision=case["precision"], mlp=bool(case.get("mlp")))
    if case.get("exact"):
        eng.set_integrator("exact")
    s = dict(case=case, eng=eng, x=x, v=v, p=_theta(case, seed), ns=ns, boxes=boxes, temps=temps)
    if k != "forces":
        s["seeds"] = systems.noise_seeds(case["steps"], seed)
    if k in ("train", "reweight"):
        s["terms"] = _targets(case, seed)
        s["loss"] = "rdf" if case["loss"] == "l2" else case["loss"]
    return s


# ------------------------------------------------------------------------------ run
def _out(case, v):
    """An engine result at the precision it has: FP32 from a mixed-precision engine."""
    return np.asarray(v, dtype=np.float32 if case["precision"] == "mixed" else np.float64)


def run(s):
    case, eng = s["case"], s["eng"]
    k = case["kind"]
    if k == "forces":
        eng.set_params(s["p"])
        eng.set_state(s["x"], s["v"])
        F = eng.forces()
        E, dE = eng.energy_grad()
        return dict(F=_out(case, F), E=E, dE=dE)
    if k == "train":
        box = s["boxes"][0] if len(s["boxes"]) == 1 else None
        sys_, lf, _ = water.forward_sim(s["x"], s["v"], box, s["seeds"], case["gamma"], case["steps"],
                                        case["every"], s["p"], 0.001, 1, case["inter"], s["loss"],
                                        loss_terms=s["terms"], engine=eng)
        back, lr, g, l_rdf, l_ev = water.reverse_sim(
            sys_.coords, sys_.velocities, box, s["seeds"], case["gamma"], case["steps"], case["every"],
            case["trunc"], s["p"], 0.001, 1, sys_.loggers, None, case["inter"], s["loss"])
        return {n: _out(case, v) for n, v in dict(
            loss=lf, v_end=sys_.velocities, loss_rev=lr, grad=g, l_rdf=l_rdf, l_ev=l_ev, x=back.coords,
            v=back.velocities).items()}
    if k == "reweight":
        sys_, l, g, l_rdf, l_ev = water.reweighting_sim(
            s["x"], s["v"], s["boxes"][0], s["seeds"], case["gamma"], case["steps"], case["every"], s["p"],
            0.001, 1, case["inter"], s["loss"], loss_terms=s["terms"], engine=eng)
        return {n: _out(case, v) for n, v in dict(loss=l, grad=g, l_rdf=l_rdf, l_ev=l_ev,
                                                  v_end=sys_.velocities).items()}
    if k == "equil":
        sys_, _, _ = water.forward_sim(s["x"], s["v"], s["boxes"][0], s["seeds"], case["gamma"], case["steps"],
                                       0, s["p"], 0.001, 1, case["inter"], "rdf", calc_loss=False,
                                       use_barostat=True, engine=eng)
        return {n: _out(case, v) for n, v in dict(box=sys_.boundary, v_end=sys_.velocities).items()}
    if k == "diamond":
        sys_, lf, *_ = sw.forward_sim(s["x"], s["v"], s["seeds"], case["gamma"], case["steps"], case["every"], 0,
                                      s["p"], s["pm"], 0.0005, engine=eng, target=s["target"])
        back, lr, g, gm = sw.reverse_sim(sys_.coords, sys_.velocities, s["seeds"], case["gamma"], case["steps"],
                                         case["every"], case["every"], 0, s["p"], s["pm"], 0.0005, 1,
                                         sys_.loggers, None)
        return {n: _out(case, v) for n, v in dict(
            loss=lf, v_end=sys_.velocities, loss_rev=lr, grad=g, grad_mlp=np.zeros(0) if gm is None else gm,
            x=back.coords, v=back.velocities).items()}
    sys_, lf, acc, _ = gas.forward_sim(s["x"], s["v"], s["seeds"], case["gamma"], case["steps"], case["every"],
                                       s["p"], 0.001, 1, case["inter"], case["loss"], engine=eng,
                                       loss_terms=s["terms"])
    v_end = sys_.velocities
    back, lr, g, Dm, l_diff, l_rdf, l_ev = gas.reverse_sim(
        sys_.coords, sys_.velocities, s["seeds"], case["gamma"], case["steps"], case["every"], case["trunc"],
        s["p"], 0.001, 1, sys_.loggers, acc, case["inter"], case["loss"])
    return {n: _out(case, v) for n, v in dict(
        loss=lf, centres=acc.gas_coords, v_end=v_end, loss_rev=lr, grad=g, D=Dm, l_diff=l_diff, l_rdf=l_rdf,
        l_ev=l_ev, v=back.velocities).items()}


# ---------------------------------------------------------------------------- exact
# The same quantities in plain torch and numpy, 64 bits, from the definitions.

C216 = 2.0 ** (1.0 / 6.0)


def _radial(form, r, p):
    """Radial pair force F(r) of the pair forms."""
    if form == "lj":
        s6 = (p[0] / r) ** 6
        return 24 * p[1] / r * (2 * s6 * s6 - s6)
    if form == "dexp":
        sig, eps, al, be = p
        rm = sig * C216
        return eps * al * be / (al - be) / rm * (torch.exp(al * (1 - r / rm)) - torch.exp(be * (1 - r / rm)))
    if form == "buck":
        return p[0] * p[1] * torch.exp(-p[1] * r) - 6 * p[2] / r ** 7
    if form == "ljsc":
        s6 = p[0] ** 6
        R = r ** 6 + s6 * p[2] * p[3] ** 2
        return 24 * p[1] * r ** 5 * (2 * s6 * s6 / R ** 3 - s6 / R ** 2)
    sig, eps, de, ga = p
    rm = sig * C216
    t = r / rm
    g7 = (1 + ga) / (t ** 7 + ga)
    b7 = ((1 + de) / (t + de)) ** 7
    return 7 * eps / rm * b7 * ((g7 - 2) / (t + de) + t ** 6 * g7 / (t ** 7 + ga))


def _pair_energy(form, r, p):
    if form == "lj":
        s6 = (p[0] / r) ** 6
        return 4 * p[1] * (s6 * s6 - s6)
    if form == "dexp":
        sig, eps, al, be = p
        t = r / (sig * C216)
        return eps * (be * torch.exp(al * (1 - t)) - al * torch.exp(be * (1 - t))) / (al - be)
    if form == "buck":
        return p[0] * torch.exp(-p[1] * r) - p[2] / r ** 6
    if form == "ljsc":
        s6 = p[0] ** 6
        q = s6 / (r ** 6 + s6 * p[2] * p[3] ** 2)
        return 4 * p[1] * (q * q - q)
    sig, eps, de, ga = p
    t = r / (sig * C216)
    return eps * ((1 + de) / (t + de)) ** 7 * ((1 + ga) / (t ** 7 + ga) - 2)


def _mlp_table(theta, nt, rc, width):
    """Cubic Hermite coefficients [nt, 1024, 4] of the learned term from its weights."""
    H, NR, NG = mlp.H, mlp.NRBF, 1024
    h = rc / NG
    r = torch.arange(NG + 1, dtype=theta.dtype, device=theta.device) * h
    mu = torch.arange(NR, dtype=theta.dtype, device=theta.device) * rc / (NR - 1)
    e = r[:, None] - mu
    phi = torch.exp(-e * e / (2 * width * width))
    dphi = -e / (width * width) * phi
    x = math.pi * r / rc
    fc, dfc = 0.5 * (torch.cos(x) + 1), -0.5 * math.pi / rc * torch.sin(x)
    out = []
    for t in range(nt):
        q = theta[t * mlp.PER_TYPE:(t + 1) * mlp.PER_TYPE]
        o = np.cumsum([0, H * NR, H, H * H, H, H, 1])
        W1, b1, W2, b2, w3, b3 = (q[o[i]:o[i + 1]] for i in range(6))
        W1, W2 = W1.view(H, NR), W2.view(H, H)

        def act(z, dz):
            s = torch.sigmoid(z)
            return z * s, s * (1 + z * (1 - s)) * dz

        a1, d1 = act(phi @ W1.T + b1, dphi @ W1.T)
        a2, d2 = act(a1 @ W2.T + b2, d1 @ W2.T)
        y, dy = a2 @ w3 + b3, d2 @ w3
        u, du = y * fc, dy * fc + y * dfc
        y0, y1, g0, g1 = u[:-1], u[1:], h * du[:-1], h * du[1:]
        out.append(torch.stack([y0, g0, 3 * (y1 - y0) - 2 * g0 - g1, 2 * (y0 - y1) + g0 + g1], 1))
    return torch.stack(out)


class _Model:
    """One periodic box of 3-site waters (and, in `gas_mol`, 2-site gas molecules, whose third
    site is an inert copy of the second): pair forces by whole-molecule neighbour tables."""

    def __init__(self, form, theta, n_mol, box, rc=C.DIST_CUTOFF, dtype=torch.float64, gas_mol=None,
                 mlp_on=False):
        self.dev, self.dtype = _device(), dtype
        self.form, self.M, self.L, self.rc = form, int(n_mol), float(box), rc
        self.krf = (78.3 - 1) / (2 * 78.3 + 1) / rc ** 3
        self.th = torch.tensor(np.asarray(theta, dtype=np.float64), dtype=dtype, device=self.dev)
        self.is_gas = torch.zeros(self.M, dtype=torch.bool, device=self.dev)
        self.has_gas = gas_mol is not None
        if self.has_gas:
            self.gas_idx = torch.tensor(np.asarray(gas_mol), device=self.dev)
            self.is_gas[self.gas_idx] = True
        nf = C.N_FORM_PARAMS[form]
        self.iq = len(C.gas_default_params(form)) - 1 if self.has_gas else nf
        qO = self.th[self.iq]
        q = torch.stack([qO, -qO / 2, -qO / 2]).expand(self.M, 3).clone()
        mass = torch.tensor([C.O_MASS, C.H_MASS, C.H_MASS], dtype=dtype, device=self.dev).expand(self.M, 3).clone()
        on = torch.tensor([True, False, False], device=self.dev).expand(self.M, 3).clone()
        if self.has_gas:
            q[self.is_gas] = 0.0
            mass[self.is_gas] = C.O_MASS
            on[self.is_gas] = torch.tensor([True, True, False], device=self.dev)
        self.q, self.mass, self.on = q, mass, on
        self.mlp_on = mlp_on
        if mlp_on:
            self.mlp_theta = self.th[nf + 5:].clone().requires_grad_(True)
            self.mlp_tab = _mlp_table(self.mlp_theta, 3, rc, 0.05)
            self.mlp_coef = self.mlp_tab.detach()
            self.mlp_adj = torch.zeros_like(self.mlp_coef)

    def class_params(self, th, c):
        """Parameters of pair class c: 0 water-water, 1 water-gas, 2 gas-gas (mixed)."""
        nf = C.N_FORM_PARAMS[self.form]
        if not self.has_gas:
            return [th[i] for i in range(nf)]
        if self.form == "buck":
            a, b = (th[:3], th[:3]) if c == 0 else (th[:3], th[3:6]) if c == 1 else (th[3:6], th[3:6])
            return [(a[i] + b[i]) / 2 for i in range(3)]
        s1, e1 = (th[0], th[1]) if c < 2 else (th[2], th[3])
        s2, e2 = (th[2], th[3]) if c > 0 else (th[0], th[1])
        return [(s1 + s2) / 2, torch.sqrt(e1 * e2)] + ([th[4], th[5]] if nf > 2 else [])

    def table(self, x, skin=0.1):
        """[M, K] partner molecules whose first sites lie within rc + skin + two bond lengths."""
        lim = (self.rc + skin + 0.25) ** 2
        o = x[:, 0]
        best, cnt = [], 0
        for c0 in range(0, self.M, 1024):
            d = o[None] - o[c0:c0 + 1024, None]
            d = d - self.L * torch.round(d / self.L)
            r2 = (d * d).sum(-1)
            i = torch.arange(c0, min(c0 + 1024, self.M), device=self.dev)
            r2[i - c0, i] = float("inf")
            ok = r2 <= lim
            cnt = max(cnt, int(ok.sum(1).max()))
            best.append(torch.where(ok, 1, 0).to(torch.int8))
        out = [torch.sort(b, dim=1, descending=True, stable=True) for b in best]
        idx = torch.cat([s.indices[:, :cnt] for s in out])
        val = torch.cat([s.values[:, :cnt] for s in out]) > 0
        return idx, val

    def mi(self, d):
        return d - self.L * torch.round(d / self.L)

    def forces_fast(self, x, tab, L):
        """Forces alone with the LJ form, no autograd, molecules in boxes of side L [M] (the
        relaxation)."""
        Lb, Lp = L[:, None], L[:, None, None]

        def mi(d, L):
            return d - L * torch.round(d / L)

        idx, val = tab
        xj, qj, onj, gj = x[idx], self.q[idx], self.on[idx], self.is_gas[idx]
        F = torch.zeros_like(x)
        b1, b2 = mi(x[:, 1] - x[:, 0], Lb), mi(x[:, 2] - x[:, 0], Lb)
        hh = mi(x[:, 2] - x[:, 1], Lb)
        w = (~self.is_gas).to(self.dtype)[:, None]

        def spring(d, k, r0):
            r = d.norm(dim=1, keepdim=True).clamp_min(1e-6)
            return k * (r - r0) * d / r

        r_hh = 2 * C.R0_BOND * math.sin(C.THETA0_ANGLE / 2)
        f1 = spring(b1, C.KB_BOND, C.R0_BOND) * w + spring(b1, C.GAS_KB_BOND, C.GAS_R0_BOND) * (1 - w)
        f2 = spring(b2, C.KB_BOND, C.R0_BOND) * w
        fh = spring(hh, 0.7e5, r_hh) * w
        F[:, 0] += f1 + f2
        F[:, 1] += fh - f1
        F[:, 2] -= f2 + fh
        for ka in range(3):
            for kb in range(3):
                d = mi(xj[:, :, kb] - x[:, None, ka], Lp)
                r2 = (d * d).sum(-1).clamp_min(0.01)
                on = val & (r2 <= self.rc * self.rc)
                i2 = 1 / r2
                A = C.COULOMB_CONST * self.q[:, None, ka] * qj[:, :, kb] * (i2 * torch.sqrt(i2) - 2 * self.krf)
                if ka < 2 and kb < 2:
                    both = self.on[:, None, ka] & onj[:, :, kb]
                    sig = torch.where(gj & self.is_gas[:, None], C.GAS_SIGMA, C.SIGMA)
                    s6 = (sig * sig * i2) ** 3
                    A = A + torch.where(both, 24 * C.EPSILON * i2 * (2 * s6 * s6 - s6), torch.zeros_like(A))
                A = torch.where(on, A, torch.zeros_like(A))
                F[:, ka] -= (A[..., None] * d).sum(1)
        return F

    def bonded_energy(self, x, th):
        w = x if not self.has_gas else x[~self.is_gas]
        if self.has_gas:
            kb, r0, ka, t0 = C.KB_BOND, C.R0_BOND, C.KA_ANGLE, C.THETA0_ANGLE
        else:
            kb, r0, ka, t0 = (th[self.iq + 1 + i] for i in range(4))
        b1, b2 = self.mi(w[:, 1] - w[:, 0]), self.mi(w[:, 2] - w[:, 0])
        r1, r2 = b1.norm(dim=1), b2.norm(dim=1)
        cth = (b1 * b2).sum(1) / (r1 * r2)
        E = 0.5 * kb * ((r1 - r0) ** 2 + (r2 - r0) ** 2).sum() + 0.5 * ka * ((torch.acos(cth) - t0) ** 2).sum()
        if self.has_gas:
            g = x[self.is_gas]
            E = E + 0.5 * C.GAS_KB_BOND * ((self.mi(g[:, 1] - g[:, 0]).norm(dim=1) - C.GAS_R0_BOND) ** 2).sum()
        return E

    def pairs_of(self, x, tab, ka, kb, c0, c1):
        idx, val = tab[0][c0:c1], tab[1][c0:c1]
        d = self.mi(x[idx][:, :, kb] - x[c0:c1, None, ka])
        r2 = (d * d).sum(-1)
        on = val & (r2 <= self.rc * self.rc)
        r = torch.sqrt(torch.where(on, r2, torch.ones_like(r2)))
        return idx, d, r, on

    def classes(self, idx, c0, c1, ka, kb, on):
        """(class, mask) of the pair-form terms of one slot."""
        if not self.has_gas:
            return [(0, on)] if ka == 0 and kb == 0 else []
        both = on & self.on[c0:c1, None, ka] & self.on[idx][:, :, kb]
        n_gas = self.is_gas[c0:c1, None].int() + self.is_gas[idx].int()
        return [(c, both & (n_gas == c)) for c in range(3)] if ka < 2 and kb < 2 else []

    def forces(self, x, tab, w=None, a=None):
        """F, and with w (and a) the VJP sum_j w_j dF_j/dx and sum a . dF/dtheta."""
        F, G = torch.zeros_like(x), torch.zeros_like(x)
        P = self.iq + 1 if self.has_gas else self.iq + 5
        dth = torch.zeros(P, dtype=self.dtype, device=self.dev)
        nc = max(1, 1_500_000 // max(1, tab[0].shape[1]))
        hinv = 1024 / self.rc
        for c0 in range(0, self.M, nc):
            c1 = min(self.M, c0 + nc)
            for ka in range(3):
                for kb in range(3):
                    idx, d, r, on = self.pairs_of(x, tab, ka, kb, c0, c1)
                    z = torch.zeros_like(r)
                    qq = C.COULOMB_CONST * self.q[c0:c1, None, ka] * self.q[idx][:, :, kb]
                    Fc = torch.where(on, qq * (1 / r ** 2 - 2 * self.krf * r), z)
                    Fr, dF = Fc.clone(), torch.where(on, -2 * qq * (1 / r ** 3 + self.krf), z)
                    na = None
                    if a is not None:
                        na = (d * a[c0:c1, None, ka]).sum(-1) / r
                        dth[self.iq] -= 2 / self.th[self.iq] * (Fc * na).sum()
                    for c, m in self.classes(idx, c0, c1, ka, kb, on):
                        rr = r[m].detach().requires_grad_(True)
                        th = self.th[:P].detach().requires_grad_(True)
                        f = _radial(self.form, rr, self.class_params(th, c))
                        df, = torch.autograd.grad(f.sum(), rr, retain_graph=a is not None)
                        Fr[m] = Fr[m] + f.detach()
                        dF[m] = dF[m] + df
                        if a is not None:
                            dth -= torch.autograd.grad((f * na[m]).sum(), th)[0]
                    if self.mlp_on:
                        t = (ka > 0) + (kb > 0)
                        q = r * hinv
                        gi = torch.clamp(q.long(), max=1023)
                        sm = q - gi
                        cf = self.mlp_coef[t][gi]
                        Fr = Fr - torch.where(on, (cf[..., 1] + sm * (2 * cf[..., 2] + 3 * sm * cf[..., 3])) * hinv, z)
                        dF = dF - torch.where(on, (2 * cf[..., 2] + 6 * sm * cf[..., 3]) * hinv * hinv, z)
                        if a is not None:
                            v = torch.where(on, na * hinv, z)
                            for k, t3 in ((1, v), (2, 2 * sm * v), (3, 3 * sm * sm * v)):
                                self.mlp_adj[t, :, k].index_add_(0, gi.reshape(-1), t3.reshape(-1))
                    A = Fr / r
                    F[c0:c1, ka] -= (A[..., None] * d).sum(1)
                    if w is not None:
                        e = w[idx][:, :, kb] - w[c0:c1, None, ka]
                        B = (dF - A) / r ** 2
                        G[c0:c1, ka] -= ((B * (d * e).sum(-1))[..., None] * d + A[..., None] * e).sum(1)
        xb = x.detach().requires_grad_(True)
        th = self.th[:P].detach().requires_grad_(True)
        g, = torch.autograd.grad(self.bonded_energy(xb, th), xb, create_graph=True)
        F -= g.detach()
        if w is not None:
            G -= torch.autograd.grad((g * w).sum(), xb, retain_graph=True)[0]
        if a is not None and not self.has_gas:
            dth -= torch.autograd.grad((g * a).sum(), th)[0]
        return F, G, dth

    def energy(self, x, tab):
        """Potential energy and its parameter gradient (without the learned term)."""
        P = self.iq + 1 if self.has_gas else self.iq + 5
        th = self.th[:P].detach().requires_grad_(True)
        E = self.bonded_energy(x, th)
        dth = torch.zeros(P, dtype=self.dtype, device=self.dev)
        if not self.has_gas:
            dth += torch.autograd.grad(E, th)[0]
        E = float(E.detach())
        shift = 1 / self.rc + self.krf * self.rc ** 2
        nc = max(1, 1_500_000 // max(1, tab[0].shape[1]))
        for c0 in range(0, self.M, nc):
            c1 = min(self.M, c0 + nc)
            for ka in range(3):
                for kb in range(3):
                    idx, _, r, on = self.pairs_of(x, tab, ka, kb, c0, c1)
                    qq = C.COULOMB_CONST * self.q[c0:c1, None, ka] * self.q[idx][:, :, kb]
                    ec = 0.5 * float(torch.where(on, qq * (1 / r + self.krf * r * r - shift), torch.zeros_like(r)).sum())
                    E += ec
                    dth[self.iq] += 2 * ec / self.th[self.iq]
                    for c, m in self.classes(idx, c0, c1, ka, kb, on):
                        e = 0.5 * _pair_energy(self.form, r[m], self.class_params(th, c)).sum()
                        E += float(e.detach())
                        dth += torch.autograd.grad(e, th)[0]
        return E, dth


def _philox(c, k0, k1):
    m32 = np.uint64(0xFFFFFFFF)
    c = [v.astype(np.uint64) for v in c]
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m32, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1),
             p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _noise(seed, n, sd):
    """The framework's documented noise: Philox4x32-10 keyed by the step seed, counter (atom,
    block), Box-Muller; sd per atom."""
    seed = int(seed)
    z = []
    for blk in (0, 1):
        a = np.arange(n, dtype=np.uint64)
        c = _philox([a, np.full(n, blk, np.uint64), np.zeros(n), np.zeros(n)], seed & 0xFFFFFFFF, seed >> 32)
        u = [((c[i] << np.uint64(21)) ^ (c[i + 1] >> np.uint64(11))) & np.uint64((1 << 53) - 1) for i in (0, 2)]
        rr = np.sqrt(-2.0 * np.log((u[0].astype(np.float64) + 1.0) / 2.0 ** 53))
        ang = 2.0 * np.pi * (u[1].astype(np.float64) / 2.0 ** 53)
        z += [rr * np.cos(ang), rr * np.sin(ang)]
    return np.stack(z[:3], 1) * np.asarray(sd)[:, None]


def _rdf(x, L, terms, grad):
    """Summed loss of the smoothed-RDF terms over water positions x [n, 3, 3] and dL/dx."""
    dev = x.device
    total, gx = 0.0, torch.zeros_like(x)
    for t in terms:
        sets = [x[:, 0] if s == 0 else x[:, 1:].reshape(-1, 3) for s in (t.sel1, t.sel2)]
        n1, n2 = len(sets[0]), len(sets[1])
        pre = L ** 3 / (4 * math.pi * n1 * n2 * t.step)
        grid = t.x_min + t.step * torch.arange(t.n_grid, dtype=x.dtype, device=dev)
        off = int(round(t.x_min / t.step)) - 1
        W = int(math.ceil(t.exp_cutoff / t.step)) + 2
        rel = torch.arange(-W, W + 1, device=dev)
        rows = max(1, 6_000_000 // (n2 * (2 * W + 1)))

        def windows(i0):
            d = sets[1][None] - sets[0][i0:i0 + rows, None]
            d = d - L * torch.round(d / L)
            r = d.norm(dim=-1)
            m = (r > 0) & (r <= t.x_min + t.step * (t.n_grid + W))
            ij = m.nonzero()
            d, r = d[m], r[m]
            k = torch.round((r - t.x_min) / t.step).long()[:, None] + rel
            xk = t.x_min + t.step * k.to(x.dtype)
            e = xk - r[:, None]
            g = torch.exp(-e * e / t.width)
            lo = torch.ceil((r - t.exp_cutoff) / t.step).long() - off - 1
            hi = torch.floor((r + t.exp_cutoff) / t.step).long() - off - 1
            ok = (k >= 0) & (k < t.n_grid)
            den = (g * (ok & (k >= lo[:, None]) & (k <= hi[:, None]))).sum(1)
            dden = (2 * e / t.width * g * (ok & (k >= lo[:, None]) & (k <= hi[:, None]))).sum(1)
            hist = ok & (r[:, None] <= xk + t.exp_cutoff) & (r[:, None] >= xk - t.exp_cutoff)
            return ij, d, r, k.clamp(0, t.n_grid - 1), e, g * hist, den, dden

        h = torch.zeros(t.n_grid, dtype=x.dtype, device=dev)
        for i0 in range(0, n1, rows):
            _, _, _, k, _, g, den, _ = windows(i0)
            v = torch.where(g.sum(1, keepdim=True) > 0, g / den[:, None], torch.zeros_like(g))
            h.index_add_(0, k.reshape(-1), v.reshape(-1))
        h = pre * h / grid ** 2
        target = torch.tensor(np.asarray(t.target, dtype=np.float64), device=dev)
        sl = t.slice_start + t.slice_stride * torch.arange(len(target), device=dev)
        e = h[sl] - target
        total += t.weight * float(e.abs().sum() if t.norm == 1 else (e * e).sum())
        if not grad:
            continue
        gh = torch.zeros_like(h)
        gh[sl] = t.weight * (torch.sign(e) if t.norm == 1 else 2 * e)
        gh = gh * pre / grid ** 2
        for i0 in range(0, n1, rows):
            ij, d, r, k, e, g, den, dden = windows(i0)
            tt = 2 * e / t.width * g / den[:, None] - g * (dden / den ** 2)[:, None]
            dl = torch.where(g.sum(1) > 0, (gh[k] * tt).sum(1), torch.zeros_like(r))
            v = (dl / r)[:, None] * d
            for s, col, sign in ((t.sel2, ij[:, 1], 1.0), (t.sel1, ij[:, 0] + i0, -1.0)):
                if s == 0:
                    gx[:, 0].index_add_(0, col, sign * v)
                else:
                    gh2 = torch.zeros(2 * len(x), 3, dtype=x.dtype, device=dev)
                    gh2.index_add_(0, col, sign * v)
                    gx[:, 1:] += gh2.view(-1, 2, 3)
    return total, gx


class _Box:
    """One box of the exact integration: flat state, masses, noise and the model's forces."""

    def __init__(self, M, sites, mass, temp, gamma, dt, seeds):
        self.M, self.sites, self.n = M, sites, len(mass)
        self.mass = torch.tensor(mass, dtype=torch.float64, device=M.dev)[:, None]
        self.sd = np.sqrt(C.KB * temp / np.asarray(mass))
        self.c = math.exp(-gamma * dt)
        self.s = math.sqrt(1 - self.c * self.c)
        self.dt, self.seeds, self.cache = dt, seeds, {}
        self.tab_age = None

    def xi(self, step):
        if self.s == 0.0:
            return 0.0
        if step not in self.cache:
            self.cache[step] = torch.tensor(_noise(self.seeds[step - 1], self.n, self.sd), device=self.M.dev)
        return self.cache[step]

    def mol(self, v):
        return v[self.sites]

    def flat(self, m):
        out = torch.zeros(self.n, 3, dtype=m.dtype, device=m.device)
        # an inert third site repeats the second: the real sites are written last
        for k in (2, 1, 0):
            out[self.sites[:, k]] = m[:, k]
        return out

    def tab(self, x, fresh=False):
        if fresh or self.tab_age is None or self.tab_age >= 20:
            self._tab, self.tab_age = self.M.table(self.mol(x)), 0
        self.tab_age += 1
        return self._tab

    def wrap(self, x):
        return x - torch.floor(x / self.M.L) * self.M.L

    def fwd(self, x, v, step):
        F = self.flat(self.M.forces(self.mol(x), self.tab(x))[0])
        v = v + F * self.dt / self.mass
        x = x + v * self.dt / 2
        v = v * self.c + self.xi(step) * self.s
        return self.wrap(x + v * self.dt / 2), v

    def back(self, x, v, g, start, n):
        """n reverse steps from step `start` with loss gradient g: (x, v, dtheta)."""
        c, dt = self.c, self.dt
        A, B = g * (1 + c), g * (1 + c)
        Cc, G = torch.zeros_like(g), torch.zeros_like(g)
        Dd = g * (1 + 2 * c + c * c) / (2 * c)
        dth = 0.0
        self.tab_age = None
        for step in range(start, start - n, -1):
            x = x - v * dt / 2
            v = (v - self.xi(step) * self.s) / c
            x = self.wrap(x - v * dt / 2)
            Dd = c * Dd + dt * dt * G * (1 + c) / 2
            Cc = Cc + Dd
            F, Gm, d = self.M.forces(self.mol(x), self.tab(x), self.mol(Cc / self.mass),
                                     self.mol(A * dt * dt / (2 * self.mass)))
            F, G = self.flat(F), self.flat(Gm)
            dth = dth + d
            v = v - F * dt / self.mass
            B = c * B + dt * dt * G
            A = A + B
        return x, v, dth


def _enth(M, x, tab, n):
    E, dE = M.energy(x, tab)
    e = C.ENTH_U_GAS - E / n + C.ENTH_RT - C.ENTH_TARGET
    return e, dE


def _water_loss(box, x, kind, terms, grad):
    """(l_rdf, l_ev, dL/dx flat, direct dl/dtheta) of one water box."""
    m = box.mol(x)
    l_rdf, gx = (0.0, torch.zeros_like(m))
    if kind in ("rdf", "both"):
        l_rdf, gx = _rdf(m, box.M.L, terms, grad)
    l_ev, dth = 0.0, 0.0
    if kind in ("enth_vap", "both"):
        tab = box.M.table(m)
        n = box.M.M
        e, dE = _enth(box.M, m, tab, n)
        l_ev, dth = e * e, -(2 * e / n) * dE
        if grad:
            gx = gx + (2 * e / n) * box.M.forces(m, tab)[0]
    return l_rdf, l_ev, box.flat(gx), dth


def _exact_train(case, s):
    outs, o = [], 0
    for r, (n, L, T) in enumerate(zip(s["ns"], s["boxes"], s["temps"])):
        n = int(n)
        M = _Model(case["inter"], s["p"], n, L, mlp_on=case["mlp"])
        sites = torch.arange(3 * n, device=M.dev).view(n, 3)
        b = _Box(M, sites, systems.masses(n), T, case["gamma"], 0.001, s["seeds"])
        x = torch.tensor(s["x"][o:o + 3 * n], device=M.dev)
        v = torch.tensor(s["v"][o:o + 3 * n], device=M.dev)
        o += 3 * n
        lf, states = 0.0, {}
        for step in range(1, case["steps"] + 1):
            x, v = b.fwd(x, v, step)
            if step % case["every"] == 0:
                lr, le, g, d = _water_loss(b, x, s["loss"], s["terms"], True)
                states[step] = (x, v, lr, le, g, d)
                lf += lr + le
        v_end, nb = v, case["steps"] // case["every"]
        l_rdf = l_ev = 0.0
        dth = 0.0
        for k in range(nb, 0, -1):
            # the blocks' ends as the reverse pass reaches them are the forward states
            xs, vs, lr, le, g, d = states[k * case["every"]]
            l_rdf, l_ev = l_rdf + lr, l_ev + le
            x, v, dd = b.back(xs, vs, g, k * case["every"], case["trunc"])
            dth = dth + dd + d
        gr = dth / nb
        if case["mlp"]:
            gm, = torch.autograd.grad((M.mlp_tab * M.mlp_adj).sum(), M.mlp_theta)
            gr = torch.cat([gr, gm / nb])
        outs.append(dict(loss=lf / nb, v_end=v_end.cpu().numpy(), loss_rev=(l_rdf + l_ev) / nb,
                         grad=gr.detach().cpu().numpy(), l_rdf=l_rdf / nb, l_ev=l_ev / nb, x=x.cpu().numpy(),
                         v=v.cpu().numpy()))
    if len(outs) == 1:
        return {k: np.asarray(v, dtype=np.float64) for k, v in outs[0].items()}
    per_atom = ("v_end", "x", "v")
    return {k: np.concatenate([q[k] for q in outs]) if k in per_atom else
            np.stack([np.asarray(q[k], dtype=np.float64) for q in outs]) for k in outs[0]}


def _exact_reweight(case, s):
    n = s["ns"][0]
    M = _Model(case["inter"], s["p"], n, s["boxes"][0])
    b = _Box(M, torch.arange(3 * n, device=M.dev).view(n, 3), systems.masses(n), C.TEMP, case["gamma"], 0.001,
             s["seeds"])
    x, v = torch.tensor(s["x"], device=M.dev), torch.tensor(s["v"], device=M.dev)
    nb = case["steps"] // case["every"]
    l = lr_ = le_ = dl = dE_ = ldE = 0.0
    for step in range(1, case["steps"] + 1):
        x, v = b.fwd(x, v, step)
        if step % case["every"] == 0:
            lr, le, _, d = _water_loss(b, x, s["loss"], s["terms"], False)
            dE = M.energy(b.mol(x), M.table(b.mol(x)))[1]
            l, lr_, le_, dl = l + lr + le, lr_ + lr, le_ + le, dl + d
            dE_, ldE = dE_ + dE, ldE + (lr + le) * dE
    g = dl / nb - (ldE / nb - (l / nb) * dE_ / nb) / (C.KB * C.TEMP)
    return {k: np.asarray(q, dtype=np.float64) for k, q in dict(
        loss=l / nb, grad=g.cpu().numpy(), l_rdf=lr_ / nb, l_ev=le_ / nb, v_end=v.cpu().numpy()).items()}


def _uniform01(seed, k):
    m = (1 << 64) - 1
    z = (seed + 0x9E3779B97F4A7C15 * (k + 1)) & m
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
    return ((z ^ (z >> 31)) >> 11) / 9007199254740992.0


def _exact_equil(case, s):
    """The barostatted run: one volume move every 30 steps, Metropolis on dU + P dV - n kT ln V'/V."""
    n = s["ns"][0]
    M = _Model(case["inter"], s["p"], n, s["boxes"][0])
    b = _Box(M, torch.arange(3 * n, device=M.dev).view(n, 3), systems.masses(n), C.TEMP, case["gamma"], 0.001,
             s["seeds"])
    x, v = torch.tensor(s["x"], device=M.dev), torch.tensor(s["v"], device=M.dev)
    seed, scale, k, kT = int(s["seeds"][0]), 0.01 * M.L ** 3, 0, C.KB * C.TEMP
    for step in range(1, case["steps"] + 1):
        x, v = b.fwd(x, v, step)
        if step % 30:
            continue
        E = M.energy(b.mol(x), M.table(b.mol(x)))[0]
        u1, u2 = _uniform01(seed, 2 * k), _uniform01(seed, 2 * k + 1)
        k += 1
        L0, V = M.L, M.L ** 3
        dV = scale * (2 * u1 - 1)
        f = ((V + dV) / V) ** (1.0 / 3.0)
        m = b.mol(x)
        h = M.mi(m - m[:, :1])
        c = m[:, :1] + h.sum(1, keepdim=True) / 3
        M.L = L0 * f
        trial = b.wrap(b.flat(m + c * f - c))
        Et = M.energy(b.mol(trial), M.table(b.mol(trial)))[0]
        dW = Et - E + 0.0602214076 * dV - n * kT * math.log((V + dV) / V)
        if dW <= 0 or u2 < math.exp(-dW / kT):
            x = trial
        else:
            M.L = L0
        b.tab_age = None
    return dict(box=np.asarray(M.L), v_end=v.cpu().numpy())


class _Sw:
    """One diamond replica: SW energy per centre over its active neighbours."""

    def __init__(self, p, pm, L):
        self.dev = _device()
        self.p = torch.tensor(p, device=self.dev)
        self.L = L
        self.coef = None
        if pm is not None:
            self.pm = torch.tensor(pm, device=self.dev).requires_grad_(True)
            self.tab = _mlp_table(self.pm, 1, D.MLP_CUTOFF, D.MLP_WIDTH)[0]
            self.coef = self.tab.detach()
            self.adj = torch.zeros_like(self.coef)

    def table(self, x, reach=0.3, K=40):
        out = []
        for c0 in range(0, len(x), 2000):
            d = x[None] - x[c0:c0 + 2000, None]
            d = d - self.L * torch.round(d / self.L)
            r2 = (d * d).sum(-1)
            i = torch.arange(c0, min(c0 + 2000, len(x)), device=self.dev)
            r2[i - c0, i] = 99.0
            out.append(torch.topk(r2, min(K, len(x) - 1), largest=False).indices)
        return torch.cat(out)

    def vectors(self, x, tab):
        d = x[tab] - x[:, None]
        d = d - self.L * torch.round(d / self.L)
        on = d.norm(dim=-1) / self.p[5] < self.p[2]
        k = int(on.sum(1).max())
        o = torch.sort(on.to(torch.int8), dim=1, descending=True, stable=True).indices[:, :k]
        return tab.gather(1, o), d.gather(1, o[..., None].expand(-1, -1, 3)), on.gather(1, o)

    def energy(self, d, on, p, coef):
        """Sum over centres of half the 2-body terms and the 3-body terms."""
        A, B, a, lam, gam, sig, eps = p
        far = torch.zeros_like(d)
        far[..., 0] = 0.5 * float(self.p[2] * self.p[5])
        d = torch.where(on[..., None], d, far)
        r = d.norm(dim=-1)
        t = 1 / (r / sig - a)
        E2 = eps * A * (B * (r / sig) ** -4 - 1) * torch.exp(t)
        E = 0.5 * torch.where(on, E2, torch.zeros_like(r)).sum()
        if coef is not None:
            q = r * (1024 / D.MLP_CUTOFF)
            g = torch.clamp(q.detach().long(), max=1023)
            s, c = q - g, coef[g]
            u = c[..., 0] + s * (c[..., 1] + s * (c[..., 2] + s * c[..., 3]))
            E = E + 0.5 * torch.where(on & (r < D.MLP_CUTOFF), u, torch.zeros_like(r)).sum()
        h = torch.where(on, torch.exp(gam * t), torch.zeros_like(r))
        u = d / r[..., None]
        cs = torch.einsum("nqa,npa->nqp", u, u) + 1.0 / 3.0
        w = torch.triu(torch.ones(h.shape[1], h.shape[1], dtype=torch.float64, device=self.dev), 1)
        return E + eps * lam * (torch.einsum("nq,np->nqp", h, h) * cs * cs * w).sum()

    def scatter(self, T, j, n):
        out = -T.sum(1)
        return out.index_add(0, j.reshape(-1), T.reshape(-1, 3))

    def grad(self, x, tab, w=None, a=None):
        """dE/dx, its derivative along w, and sum a . d(dE/dx)/dtheta."""
        j, d, on = self.vectors(x, tab)
        d = d.detach().requires_grad_(True)
        p = self.p.detach().requires_grad_(True)
        cf = None if self.coef is None else self.coef.detach().requires_grad_(True)
        T, = torch.autograd.grad(self.energy(d, on, p, cf), d, create_graph=w is not None)
        g = self.scatter(T.detach(), j, len(x))
        if w is None:
            return g, None, None
        Tt, = torch.autograd.grad((T * (w[j] - w[:, None])).sum(), d, retain_graph=True)
        z = a[j] - a[:, None]
        th = torch.autograd.grad((T * z).sum(), [p] + ([] if cf is None else [cf]))
        if cf is not None:
            self.adj -= th[1]
        return g, self.scatter(Tt, j, len(x)), th[0]

    def loss(self, x, v, tab, target, weight=D.STRESS_WEIGHT):
        """Stress loss, dL/dx, dL/dv and dL/dtheta (the learned term's into adj)."""
        V = self.L ** 3
        j, d, on = self.vectors(x, tab)
        d = d.detach().requires_grad_(True)
        p = self.p.detach().requires_grad_(True)
        cf = None if self.coef is None else self.coef.detach().requires_grad_(True)
        T, = torch.autograd.grad(self.energy(d, on, p, cf), d, create_graph=True)
        vv = v.detach().requires_grad_(True)
        dv = vv - vv.mean(0)
        sig = (torch.einsum("nqa,nqb->ab", T, d) - D.C_MASS * dv.T @ dv) / V
        l = weight * ((sig - target) ** 2).sum() / 9
        gr = torch.autograd.grad(l, [d, vv, p] + ([] if cf is None else [cf]))
        if cf is not None:
            self.adj += gr[3]
        return float(l.detach()), self.scatter(gr[0], j, len(x)), gr[1], gr[2]


def _exact_diamond(case, s):
    R, n, dt, gamma = case["reps"], 8 * case["cells"] ** 3, 0.0005, case["gamma"]
    c = math.exp(-gamma * dt)
    sn, m = math.sqrt(1 - math.exp(-2 * gamma * dt)), D.C_MASS
    sd = np.full(n, math.sqrt(D.KB * D.TEMP / m))
    noise = [_noise(q, n, sd) for q in s["seeds"]]
    outs = []
    for r in range(R):
        S = _Sw(s["p"], s["pm"], s["box"])
        xi = [torch.tensor(q, device=S.dev) for q in noise]
        target = torch.tensor(s["target"], device=S.dev)
        x = torch.tensor(s["x"][r * n:(r + 1) * n], device=S.dev)
        v = torch.tensor(s["v"][r * n:(r + 1) * n], device=S.dev)
        tab = S.table(x)
        wrap = lambda q: q - torch.floor(q / s["box"]) * s["box"]  # noqa: E731
        ends = {}
        for step in range(1, case["steps"] + 1):
            v = v - S.grad(x, tab)[0] * dt / m
            x = x + v * dt / 2
            v = v * c + xi[step - 1] * sn
            x = wrap(x + v * dt / 2)
            if (case["steps"] - step) % case["every"] == 0:
                ends[step] = (x, v)
        v_end, nb, l, gp = v, len(ends), 0.0, 0.0
        for k in sorted(ends, reverse=True):
            x, v = ends[k]
            lk, gx, gv, gt = S.loss(x, v, tab, target)
            l, gp = l + lk, gp + gt
            A = gx * (1 + c) + gv * c * 2 / dt
            B = gx * (1 + c) + gv * (c - 1) * 2 / dt
            Cc = gv * (1 + c) / dt
            Dd = gx * (1 + 2 * c + c * c) / (2 * c) + gv * (c - 1 / c) / dt
            G = torch.zeros_like(gx)
            for step in range(k, max(k - case["every"], 0), -1):
                x = x - v * dt / 2
                v = (v - xi[step - 1] * sn) / c
                x = wrap(x - v * dt / 2)
                Dd = c * Dd + dt * dt * G * (1 + c) / 2
                Cc = Cc + Dd
                g, gt, th = S.grad(x, tab, Cc / m, A * dt * dt / (2 * m))
                G = -gt
                gp = gp - th
                v = v + g * dt / m
                B = c * B + dt * dt * G
                A = A + B
        gm = np.zeros(0)
        if S.coef is not None:
            gm = torch.autograd.grad((S.tab * S.adj).sum(), S.pm)[0].cpu().numpy() / nb
        outs.append(dict(loss=l / nb, v_end=v_end.cpu().numpy(), grad=(gp / nb).cpu().numpy(), grad_mlp=gm,
                         x=x.cpu().numpy(), v=v.cpu().numpy()))
    cat, mean = (lambda k: np.concatenate([q[k] for q in outs])), (lambda k: np.mean([q[k] for q in outs], axis=0))
    return dict(loss=np.asarray(mean("loss")), v_end=cat("v_end"), loss_rev=np.asarray(mean("loss")),
                grad=mean("grad"), grad_mlp=mean("grad_mlp"), x=cat("x"), v=cat("v"))


def _diffusion(gc, L, lf):
    """Diffusion coefficient (nm^2/ps) of the unwrapped gas centres gc [frames, n_gas, 3]."""
    ns = gc.shape[0] // 2
    Dv = 0.0
    for f in range(ns):
        t = gc[f]
        for j in range(f + 1, f + ns + 1):
            d = gc[j] - t
            t = t + d - L * torch.round(d / L)
        Dv = Dv + ((t - gc[f]) ** 2).sum(1).mean() / (ns * lf)
    return Dv / (6 * ns)


def _exact_gas(case, s):
    nw, ng, L, dt = case["n_water"], case["n_gas"], case["box"], 0.001
    n = nw + ng
    M = _Model(case["inter"], s["p"], n, L, gas_mol=np.arange(nw, n))
    w = np.arange(3 * nw).reshape(nw, 3)
    o = 3 * nw + 2 * np.arange(ng)
    sites = torch.tensor(np.concatenate([w, np.stack([o, o + 1, o + 1], 1)]), device=M.dev)
    b = _Box(M, sites, systems.gas_water_masses(nw, ng), C.TEMP, case["gamma"], dt, s["seeds"])
    x, v = torch.tensor(s["x"], device=M.dev), torch.tensor(s["v"], device=M.dev)
    nb, ends = case["steps"] // case["every"], {}
    for step in range(1, case["steps"] + 1):
        x, v = b.fwd(x, v, step)
        if step % case["every"] == 0:
            ends[step // case["every"]] = (x, v)
    v_end = v
    cent = []
    for k in range(1, nb + 1):
        g = ends[k][0][3 * nw:].view(ng, 2, 3)
        q = g[:, 0] + M.mi(g[:, 1] - g[:, 0]) / 2
        cent.append(q - torch.floor(q / L) * L)
    gc = torch.stack(cent).requires_grad_(True)
    Dv = _diffusion(gc, L, case["every"] * dt)
    dgc, = torch.autograd.grad(Dv, gc)
    Dm = float(Dv.detach()) * 1e-6
    l_diff = 1e18 * (Dm - 2e-9) ** 2
    dgc = dgc * (1e18 * 2 * (Dm - 2e-9) * 1e-6)
    dth, l_rdf, l_ev = 0.0, 0.0, 0.0
    for k in range(nb, 0, -1):
        xs, vs = ends[k]
        m = b.mol(xs)
        gx = torch.zeros_like(xs)
        if "ev" in case["loss"]:
            tab = M.table(m)
            e, dE = _enth(M, m, tab, n)
            kk = 2 * e * 0.05 / (nb * n)
            l_ev += 0.05 * e * e / nb
            gx += kk * b.flat(M.forces(m, tab)[0])
            dth = dth - kk * dE
        if "rdf" in case["loss"]:
            lr, gw = _rdf(m[:nw], L, s["terms"], True)
            l_rdf += 0.05 * lr / nb
            gx[:3 * nw] += 0.05 / nb * gw.reshape(-1, 3)
        gx[3 * nw:] += (dgc[k - 1] / 2).repeat_interleave(2, 0)
        x, v, dd = b.back(xs, vs, gx, k * case["every"], case["trunc"])
        dth = dth + dd
    tot = l_diff + l_rdf + l_ev
    return {k: np.asarray(q, dtype=np.float64) for k, q in dict(
        loss=tot, centres=gc.detach().cpu().numpy(), v_end=v_end.cpu().numpy(), loss_rev=tot,
        grad=dth.cpu().numpy(), D=Dm, l_diff=l_diff, l_rdf=l_rdf, l_ev=l_ev, v=v.cpu().numpy()).items()}


def exact(case, seed):
    """What run() returns for these inputs, in 64 bits from the definitions."""
    s = prepare(case, seed)
    s["eng"].close()
    k = case["kind"]
    if k == "forces":
        n = s["ns"][0]
        M = _Model(case["inter"], s["p"], n, s["boxes"][0])
        x = torch.tensor(s["x"], device=M.dev).view(n, 3, 3)
        tab = M.table(x)
        E, dE = M.energy(x, tab)
        return dict(F=M.forces(x, tab)[0].reshape(-1, 3).cpu().numpy(), E=np.array([E]), dE=dE.cpu().numpy()[None])
    return dict(train=_exact_train, reweight=_exact_reweight, equil=_exact_equil, diamond=_exact_diamond,
                gas=_exact_gas)[k](case, s)
