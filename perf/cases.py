"""Timed cases of the force path and the error-estimate tools, through the public Python API.

A case is a dict of plain values; prepare() makes what a program holds before the call (systems,
lists, engines, meshes, handles), run() is one pass, exact() the same results from plain torch in
64 bits.  Kinds:

  md       Simulation.run(steps) and the frame (positions, velocities) read afterwards
  forces   forces of new positions from device memory: cell sort, neighbour list, pair forces and,
           with charges, real-space Ewald and SPME
  grad     SPME energy with its gradient by torch.autograd
  hermite  energy and force-error functional of candidate Hermite bases with every gradient
  arc      one adaptive-cutoff update of a density sample
  errmap   the ik-SPME error map of one choice of (beta, mesh)
  ikerr    the optiBasis functional of a batch of candidate bases with its gradient
  ewald    the exact reciprocal Ewald sum

Results of a mixed-precision system are binary32 numbers carried in 64-bit arrays by the API; the
program keeps them as float32.  Positions and boxes are binary32 values, so both precisions see
the same system.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "md.error_b200"))

import mdforce as mdf  # noqa: E402

DT, SKIN_FLUID, SKIN_SLAB, CELL = 0.005, 0.3, 0.6, 2.8
ORDER = 6


def listed():
    return [
        # the 4,000-atom LJ fluid: the smallest system run in earnest, where latency and launches count
        {"name": "md_lj_fluid_4k", "kind": "md", "shape": "fluid", "n": 4000, "charged": False, "mixed": True,
         "rc": 2.5, "steps": 50},
        # the headline workload: the 65,536-atom liquid-vapour slab, Langevin NPT along z, adaptive cutoffs
        # re-estimated on the reference's schedule
        {"name": "md_lj_slab_64k", "kind": "md", "shape": "slab", "n": 65536, "charged": False, "mixed": True,
         "rc": 5.0, "steps": 40},
        # the 20,736-charge fluid with the full Ewald split every step
        {"name": "md_charged_fluid_20k", "kind": "md", "shape": "fluid", "n": 20736, "charged": True, "mixed": True,
         "rc": 3.0, "steps": 20},
        # forces of one configuration in plain FP64 (reference forces of the error studies, or an external integrator)
        {"name": "forces_lj_slab_64k_fp64", "kind": "forces", "shape": "slab", "n": 65536, "charged": False,
         "mixed": False, "rc": 5.0, "method": "ik"},
        # the LJ + SPME slab: list, real space and the reciprocal chain on 128 x 128 x 512, mixed precision
        {"name": "forces_charged_slab_64k", "kind": "forces", "shape": "slab", "n": 65536, "charged": True,
         "mixed": True, "rc": 5.0, "method": "ik"},
        # energy and gradient of the charged fluid in FP64, forward and backward, as an optimiser calls it
        {"name": "grad_fluid_20k_fp64", "kind": "grad", "shape": "fluid", "n": 20736, "mixed": False},
        # the same for the million-charge slab on 128 x 128 x 512 in mixed precision: the largest system
        {"name": "grad_slab_1m", "kind": "grad", "shape": "slab", "n": 1048576, "mixed": True},
        # one optimisation step over 8 candidate bases of order-6 support on the charged fluid
        {"name": "hermite_8x20k", "kind": "hermite", "n": 20736, "cand": 8, "half": 3, "nbin": 16},
        # the cutoff update of the slab run, 41 x 41 x 161 bins, cutoffs 2.5 to 5.0
        {"name": "adapt_rcut_slab_64k", "kind": "arc", "n": 65536},
        # one candidate (beta, mesh) of a parameter choice: kernel, profile and RMS map
        {"name": "error_map_64", "kind": "errmap", "n": 20736, "k0": 64, "k1": 64, "k2": 64, "order": 6},
        # the functional that optiBasis minimises, value and gradient of 8 candidates
        {"name": "ik_error_8", "kind": "ikerr", "cand": 8, "k": 64, "nbin": 16},
        # exact reciprocal sum of a small charged system, the yardstick of the SPME errors
        {"name": "ewald_exact_4k", "kind": "ewald", "n": 4000, "k": 32},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["md", "md", "forces", "forces", "grad", "hermite", "arc", "errmap", "ikerr", "ewald"])
    shape = rng.choice(["fluid", "slab"])
    mixed = rng.random() < 0.6
    if kind == "md":
        charged = rng.random() < 0.5
        n = _log(rng, 4096 if shape == "slab" else 1500, 24000 if charged else 65536)
        return {"kind": kind, "shape": shape, "n": n, "charged": charged, "mixed": mixed,
                "rc": 5.0 if shape == "slab" else rng.choice([2.5, 3.0, 3.5]), "steps": rng.randint(10, 20 if charged else 40)}
    if kind == "forces":
        charged = rng.random() < 0.5
        return {"kind": kind, "shape": shape, "n": _log(rng, 4096 if shape == "slab" else 1500, 65536),
                "charged": charged, "mixed": mixed, "rc": 5.0 if shape == "slab" else rng.choice([2.5, 3.0, 3.5]),
                "method": rng.choice(["ik", "analytic"])}
    if kind == "grad":
        return {"kind": kind, "shape": shape, "n": _log(rng, 2000, 500000 if mixed else 120000), "mixed": mixed}
    if kind == "hermite":
        return {"kind": kind, "n": _log(rng, 1500, 20736), "cand": rng.randint(1, 8), "half": rng.choice([2, 3]),
                "nbin": rng.choice([8, 12, 16])}
    if kind == "arc":
        return {"kind": kind, "n": _log(rng, 4096, 65536)}
    if kind == "errmap":
        return {"kind": kind, "n": _log(rng, 1500, 20736), "k0": rng.randint(16, 64), "k1": rng.choice([16, 32, 64]),
                "k2": rng.randint(16, 64), "order": rng.choice([4, 5, 6])}
    if kind == "ikerr":
        return {"kind": kind, "cand": rng.randint(1, 16), "k": rng.choice([32, 48, 64, 96, 128]),
                "nbin": rng.choice([8, 12, 16])}
    return {"kind": "ewald", "n": _log(rng, 300, 4000), "k": rng.randint(8, 32)}


# ---------------------------------------------------------------- systems
class _System:
    """Positions, velocities, charges and box of a seeded fluid or liquid-vapour slab."""

    def __init__(self, shape, n, charged, seed):
        rng = np.random.default_rng([seed & 0xffffffff, n])
        if shape == "fluid":
            # fcc sites (vacancies where n is no whole crystal) with a thermal spread, density 0.8
            edge = float(np.float32((n / 0.8) ** (1.0 / 3.0)))
            nc = math.ceil((n / 4.0) ** (1.0 / 3.0) - 1e-9)
            box = np.array([edge, edge, edge])
            pos = _fcc((nc, nc, nc), box)[rng.permutation(4 * nc ** 3)[:n]]
            spread, self.temp = 0.04 * edge / nc, 1.0
        else:
            # liquid at 0.78 in the middle of a box of 1 : 1 : 4, vapour at 0.02 on a coarse random grid around it
            edge = float(np.float32(40.0 * (n / 65536.0) ** (1.0 / 3.0)))
            box = np.array([edge, edge, float(np.float32(4.0 * edge))])
            thick = (n - 0.02 * box.prod()) / (0.76 * edge * edge)
            nx = max(1, round(edge / 1.7242))
            az = 4.0 / (0.78 * (edge / nx) ** 2)
            n_liq = int(round(0.78 * edge * edge * thick))
            nz = math.ceil(n_liq / (4.0 * nx * nx))
            liq = _fcc((nx, nx, nz), np.array([edge, edge, az * nz]))
            liq[:, 2] += 0.5 * (box[2] - az * nz)
            liq = liq[np.argsort(np.abs(liq[:, 2] - 0.5 * box[2]), kind="stable")[:n_liq]]
            free = np.abs(liq[:, 2] - 0.5 * box[2]).max() + 1.3
            g = [max(1, int(box[0] / 2.4)), max(1, int(box[1] / 2.4))]
            gz = max(1, int((box[2] - 2 * free) / 2.4))
            ix = rng.permutation(g[0] * g[1] * gz)[:n - n_liq]
            vap = np.stack([(ix // (g[1] * gz) + 0.5) * box[0] / g[0], (ix // gz % g[1] + 0.5) * box[1] / g[1],
                            0.5 * box[2] + free + (ix % gz + 0.5) * (box[2] - 2 * free) / gz], 1)
            pos = np.concatenate([liq, vap])[rng.permutation(n)]
            spread, self.temp = 0.07, 0.85
        pos = pos + np.clip(rng.normal(0.0, spread, pos.shape), -2.5 * spread, 2.5 * spread)
        pos = np.mod(pos, box).astype(np.float32).astype(np.float64)
        pos[pos >= box] = 0.0
        self.pos, self.box, self.n = pos, box, n
        self.vel = rng.normal(0.0, math.sqrt(self.temp), pos.shape).astype(np.float32).astype(np.float64)
        self.vel -= self.vel.mean(0)
        self.charge = None
        if charged:
            self.charge = np.zeros(n)
            self.charge[rng.permutation(n)[:n - n % 2]] = np.tile([1.0, -1.0], n // 2)
        # cutoffs of the slab by region as the estimate assigns them: 4.0 in the liquid, 5.0 at the
        # interfaces, 2.5 to 3.0 in the vapour
        nb = [int(b) | 1 for b in box]
        z = (np.arange(nb[2]) + 0.5) * box[2] / nb[2] - 0.5 * box[2]
        half = 0.5 * n / (0.78 * box[0] * box[1])
        rc = np.where(np.abs(np.abs(z) - half) < 3.5, 5.0, np.where(np.abs(z) < half, 4.0, 3.0))
        lat = np.broadcast_to(rc, nb).astype(np.float32)
        self.lattice = np.where((lat == 3.0) & (rng.random(nb) < 0.2) & (not charged), np.float32(2.5), lat)
        # mesh spacing of about a third to a half, powers of two; splitting for the smallest cutoff
        self.mesh = tuple(1 << max(3, round(math.log2(b / 0.4))) for b in box)
        self.beta = 0.95


def _fcc(cells, box):
    base = np.array([[0.25, 0.25, 0.25], [0.75, 0.75, 0.25], [0.75, 0.25, 0.75], [0.25, 0.75, 0.75]])
    i = np.stack(np.meshgrid(*[np.arange(c) for c in cells], indexing="ij"), -1).reshape(-1, 1, 3)
    return ((i + base) / np.array(cells)).reshape(-1, 3) * box


def _of(case, seed):
    return _System(case.get("shape", "fluid"), case["n"], case.get("charged", case["kind"] in
                   ("grad", "hermite", "errmap", "ewald")), seed)


def _cutoffs(case, s, sys_):
    if case["shape"] == "slab":
        mdf.AssignRCut(s.lattice).assign(sys_)
    else:
        sys_.set_rcut(np.full(s.n, case["rc"], np.float32))


def _candidates(cand, half, nbin, seed):
    base = mdf.optibasis.bspline_initial_basis(float(half), nbin, 2 * half)
    g = torch.Generator().manual_seed(seed)
    c = torch.from_numpy(np.tile(base, (cand, 1)))
    return (c * (1.0 + 0.02 * torch.randn(c.shape, generator=g, dtype=torch.float64))).cuda()


# ---------------------------------------------------------------- prepare
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return globals()["_run_" + state["kind"]](state)


def _prepare_md(case, seed):
    s = _of(case, seed)
    sys_ = mdf.MDSystem(s.pos, s.box, vel=s.vel, charge=s.charge, precision=mdf.PREC_MIXED if case["mixed"] else mdf.PREC_FP64)
    _cutoffs(case, s, sys_)
    eng = mdf.InteractionEngine(sys_)
    eng.registNonBondedInteraction(1.0, 1.0, 0.0)
    spme = None
    if case["charged"]:
        mdf.registCoulomb(eng, s.beta)
        spme = mdf.SPME(sys_, s.mesh, ORDER, s.beta)
    slab = case["shape"] == "slab"
    lv = mdf.langevin_params(dt=DT, temperature=s.temp, gamma_t=1.0, tau_p=2.0, kappa_t=0.1, npt_dirs=4 if slab else 0,
                             seed=1 + seed % 1000003)
    sim = mdf.Simulation(sys_, eng, skin=SKIN_SLAB if slab else SKIN_FLUID, cell_size=CELL, lv=lv,
                         max_rcut=case["rc"], spme=spme)
    if slab and not case["charged"]:
        arc = mdf.AdaptRCutEstimator(sys_, refh=1.0, rcmin=2.5, rcmax=5.0, rcstep=0.5)
        sim.attach_adapt_rcut(arc, sample_every=40, update_every=2000, prec=0.02)
    return {"kind": "md", "sys": sys_, "sim": sim, "steps": case["steps"], "mixed": case["mixed"]}


def _kept(a, mixed):
    return a.astype(np.float32) if mixed else a


def _run_md(st):
    st["sim"].run(st["steps"])
    return {"positions": _kept(st["sys"].unwrapped_positions(), st["mixed"]),
            "velocities": _kept(st["sys"].velocities(), st["mixed"])}


def _prepare_forces(case, seed):
    s = _of(case, seed)
    sys_ = mdf.MDSystem(s.pos, s.box, charge=s.charge, precision=mdf.PREC_MIXED if case["mixed"] else mdf.PREC_FP64)
    _cutoffs(case, s, sys_)
    eng = mdf.InteractionEngine(sys_)
    eng.registNonBondedInteraction(1.0, 1.0, 0.0)
    spme = None
    if case["charged"]:
        mdf.registCoulomb(eng, s.beta)
        spme = mdf.SPME(sys_, s.mesh, ORDER, s.beta, method=case["method"])
    cl = mdf.CellList(sys_, CELL)
    cl.rebuild()
    nl = mdf.NeighborList(sys_, case["rc"], 0.0, expansion=1.5)
    nl.fit(sys_, cl)
    sys_.set_stream(torch.cuda.current_stream().cuda_stream)
    return {"kind": "forces", "sys": sys_, "eng": eng, "spme": spme, "cl": cl, "nl": nl, "mixed": case["mixed"],
            "pos": torch.tensor(s.pos, device="cuda")}


def _run_forces(st):
    sys_ = st["sys"]
    sys_.set_device_view(pos_ptr=st["pos"].data_ptr())
    st["cl"].rebuild(sys_)
    st["nl"].rebuild(sys_, st["cl"])
    st["eng"].clearInteraction(sys_)
    st["eng"].applyNonBondedInteraction(sys_, st["nl"])
    if st["spme"] is not None:
        st["spme"].apply(sys_)
    return _kept(sys_.forces(), st["mixed"])


def _grad_system(case, seed):
    s = _of(case, seed)
    if case["shape"] == "slab" and case["n"] > 400000:
        s.mesh = (128, 128, 512)
    return s


def _prepare_grad(case, seed):
    s = _grad_system(case, seed)
    sys_ = mdf.MDSystem(s.pos, s.box, charge=s.charge, precision=mdf.PREC_MIXED if case["mixed"] else mdf.PREC_FP64)
    cl = mdf.CellList(sys_, CELL)
    cl.rebuild()
    spme = mdf.SPME(sys_, s.mesh, ORDER, s.beta)
    return {"kind": "grad", "spme": spme, "cl": cl, "mixed": case["mixed"],
            "q": torch.tensor(s.charge, device="cuda", requires_grad=True),
            "r": torch.tensor(s.pos, device="cuda", requires_grad=True)}


def _run_grad(st):
    q, r = st["q"], st["r"]
    q.grad = r.grad = None
    e = mdf.optibasis.spme_energy(q, r, st["spme"])
    e.backward()
    out = {"energy": e.detach(), "dq": q.grad, "dr": r.grad}
    return {k: v.float() for k, v in out.items()} if st["mixed"] else out


def _prepare_hermite(case, seed):
    s = _of(case, seed)
    g = torch.Generator().manual_seed(seed)
    return {"kind": "hermite", "hs": mdf.optibasis.HermiteSPME(s.n, s.mesh, s.box, s.beta, float(case["half"]), case["nbin"]),
            "q": torch.tensor(s.charge, device="cuda"), "r": torch.tensor(s.pos, device="cuda"),
            "c": _candidates(case["cand"], case["half"], case["nbin"], seed),
            "fref": (0.3 * torch.randn(s.n, 3, generator=g, dtype=torch.float64)).cuda()}


def _run_hermite(st):
    a = st["hs"].energy(st["q"], st["r"], st["c"], forces=True, grads=True)
    b = st["hs"].force_error(st["q"], st["r"], st["c"], st["fref"], grads=True)
    return [a, b]


def _prepare_arc(case, seed):
    s = _System("slab", case["n"], False, seed)
    sys_ = mdf.MDSystem(s.pos, s.box)
    sys_.set_stream(torch.cuda.current_stream().cuda_stream)
    arc = mdf.AdaptRCutEstimator(sys_, refh=1.0, rcmin=2.5, rcmax=5.0, rcstep=0.5)
    # the samples gathered since the last update: displaced frames, as a run deposits them
    g = torch.Generator(device="cuda").manual_seed(seed)
    pos, box = torch.tensor(s.pos, device="cuda"), torch.tensor(s.box, device="cuda")
    for _ in range(24):
        move = box * torch.rand(3, generator=g, dtype=torch.float64, device="cuda")
        move[2] = 0.0
        frame = torch.remainder(pos + move + 0.5 * torch.randn(pos.shape, generator=g, dtype=torch.float64, device="cuda"),
                                box)
        sys_.set_device_view(pos_ptr=frame.data_ptr())
        arc.deposite()
    return {"kind": "arc", "sys": sys_, "arc": arc}


def _run_arc(st):
    # the last sample, the new cutoff map, and the map written out
    arc = st["arc"]
    arc.deposite()
    arc.update(0.02)
    arc.assign()
    rc, idx, err = arc.rcut()
    return {"rc": rc, "index": idx, "error": err}


def _prepare_errmap(case, seed):
    s = _of(case, seed)
    return {"kind": "errmap", "sys": mdf.MDSystem(s.pos, s.box, charge=s.charge, precision=mdf.PREC_FP64),
            "box": s.box, "beta": s.beta, "K": (case["k0"], case["k1"], case["k2"]), "order": case["order"]}


def _run_errmap(st):
    em = mdf.ErrorEstimate_SPME_Ik(st["K"], st["box"], st["beta"], st["order"])
    em.deposit(st["sys"])
    return em.rms(1.0)


def _prepare_ikerr(case, seed):
    return {"kind": "ikerr", "f": mdf.optibasis.HermiteLossFunc(2.0, case["nbin"], 0.95, [case["k"]] * 3, 20736.0, 20736,
                                                                [30.0, 30.0, 30.0]),
            "x": _candidates(case["cand"], 2, case["nbin"], seed).requires_grad_(True)}


def _run_ikerr(st):
    x = st["x"]
    x.grad = None
    loss = mdf.optibasis.ik_error_loss(x, st["f"])
    loss.sum().backward()
    return {"loss": loss.detach(), "grad": x.grad}


def _prepare_ewald(case, seed):
    s = _of(case, seed)
    sys_ = mdf.MDSystem(s.pos, s.box, charge=s.charge, precision=mdf.PREC_FP64)
    return {"kind": "ewald", "sys": sys_, "eng": mdf.InteractionEngine(sys_), "K": (case["k"],) * 3, "beta": s.beta}


def _run_ewald(st):
    st["eng"].clearInteraction()
    e = mdf.ewald_exact(st["sys"], st["K"], st["beta"])
    return {"energy": e, "forces": st["sys"].forces()}


# ---------------------------------------------------------------- work
def work(case):
    """Bytes: inputs and outputs of the pass once (for md, the state once per step).  Operations: the
    pair terms within the cutoffs, stencils, 5 n log2 n per transform."""
    n, kind = case.get("n", 0), case["kind"]
    if kind == "ikerr":
        kmax, nc = case["k"] * 10.5 + 1, 2 * case["nbin"]
        return {"bytes": 8.0 * (3 * (1 + nc) * kmax + 2 * case["cand"] * nc),
                "flops": 3.0 * case["cand"] * nc * kmax * 4}
    if kind == "ewald":
        nm = (2 * (case["k"] // 2) + 1) ** 3
        return {"bytes": 56.0 * n, "flops": 0.5 * nm * n * 20}
    if kind == "errmap":
        K = case["k0"] * case["k1"] * case["k2"]
        return {"bytes": 32.0 * n + 8.0 * K, "flops": 5.0 * K * math.log2(K) * 32}
    shape = "slab" if kind == "arc" else case.get("shape", "fluid")
    edge = (n / 0.8) ** (1 / 3) if shape == "fluid" else 40.0 * (n / 65536.0) ** (1 / 3)
    box = (edge, edge, edge if shape == "fluid" else 4 * edge)
    if kind == "arc":
        K = math.prod(int(b) | 1 for b in box)
        return {"bytes": 16.0 * n + 8.0 * K * (6 * 7 + 3), "flops": 5.0 * K * math.log2(K) * 25}
    mesh = (128, 128, 512) if kind == "grad" and shape == "slab" and n > 400000 else \
        tuple(1 << max(3, round(math.log2(b / 0.4))) for b in box)
    K = math.prod(mesh)
    fft = 2.5 * K * math.log2(K)
    if kind == "hermite":
        c, pts = case["cand"], 8 * case["half"] ** 3
        return {"bytes": 8.0 * n * (7 + 11 * c), "flops": c * (n * pts * 60.0 + 13 * fft)}
    el = 4.0 if case["mixed"] else 8.0
    if kind == "grad":
        return {"bytes": 8.0 * n * 8, "flops": n * ORDER ** 3 * 12.0 + 2 * fft}
    rc = case["rc"] if shape == "fluid" else 4.1
    pairs = n * 4.19 * rc ** 3 * 0.78
    flops = pairs * (40.0 if case["charged"] else 20.0) + case["charged"] * (n * ORDER ** 3 * 10.0 + 4 * fft)
    if kind == "md":
        return {"bytes": case["steps"] * n * 16 * el, "flops": case["steps"] * (flops + 100.0 * n)}
    return {"bytes": 48.0 * n, "flops": flops}


# ---------------------------------------------------------------- exact
def exact(case, seed):
    fn = globals().get("_exact_" + case["kind"])
    # md: a trajectory has no value apart from the driver's own noise stream; arc: the estimate's kernels are
    # defined by an adaptive quadrature at the reference's own tolerances, not by the integrals' values
    return None if fn is None else fn(case, seed)


def _cuda(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _rcut_of(case, s):
    if case["shape"] != "slab":
        return torch.full((s.n,), case["rc"], dtype=torch.float64, device="cuda")
    n, ix = s.lattice.shape, []
    for d in range(3):
        x = s.pos[:, d].astype(np.float32) * np.float32(n[d]) / np.float32(s.box[d])
        ix.append(np.clip(x.astype(np.int64), 0, n[d] - 1))
    return _cuda(s.lattice[tuple(ix)].astype(np.float64))


def _exact_forces(case, seed):
    s = _of(case, seed)
    x, L, rc = _cuda(s.pos), s.box, _rcut_of(case, s)
    q = None if s.charge is None else _cuda(s.charge)
    F = torch.zeros_like(x)
    step = max(1, (1 << 25) // s.n)
    for i in range(0, s.n, step):
        d = [x[i:i + step, k:k + 1] - x[None, :, k] for k in range(3)]
        d = [a - L[k] * torch.floor(a / L[k] + 0.5) for k, a in enumerate(d)]
        r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
        on = r2 < (rc[i:i + step] ** 2)[:, None]
        on[torch.arange(on.shape[0], device="cuda"), torch.arange(i, i + on.shape[0], device="cuda")] = False
        r2 = torch.where(on, r2, 1e30)
        s6 = 1.0 / r2 ** 3
        f = 24.0 * (2.0 * s6 * s6 - s6) / r2
        if q is not None:
            r = r2.sqrt()
            f = f + q[i:i + step, None] * q[None, :] * (torch.erfc(s.beta * r) / r + 2.0 * s.beta / math.sqrt(math.pi) *
                                                         torch.exp(-s.beta ** 2 * r2)) / r2
        F[i:i + step] = torch.stack([(f * a).sum(1) for a in d], 1)
    if q is not None:
        F = F + _spme(s, q, x, case["method"])["force"]
    return F.cpu().numpy()


def _weights(f):
    """M_n(f + j), j = 0..n-1, and the derivatives of the cardinal B-spline of order ORDER: two [n] lists."""
    w = [f, 1.0 - f]
    for k in range(3, ORDER + 1):
        prev = w + [torch.zeros_like(f)]
        if k == ORDER:
            dw = [prev[j] - (prev[j - 1] if j else 0.0) for j in range(ORDER)]
        w = [((f + j) * prev[j] + (k - f - j) * (prev[j - 1] if j else 0.0)) / (k - 1) for j in range(k)]
    return w, dw


def _spme(s, q, x, method):
    """SPME of charges q at x: energy, and the force of the differentiation method, or (method None) the gradient."""
    K, L, V = s.mesh, s.box, float(np.prod(s.box))
    idx, W, D = [], [], []
    for d in range(3):
        u = torch.remainder(x[:, d] * (K[d] / L[d]), K[d])
        b = torch.floor(u)
        w, dw = _weights(u - b)
        W.append(w)
        D.append(dw)
        idx.append([torch.remainder(b.long() - j, K[d]) for j in range(ORDER)])
    stencil = [(a, b, c) for a in range(ORDER) for b in range(ORDER) for c in range(ORDER)]

    def at(p):
        return (idx[0][p[0]] * K[1] + idx[1][p[1]]) * K[2] + idx[2][p[2]]

    Q = torch.zeros(K[0] * K[1] * K[2], dtype=torch.float64, device="cuda")
    for p in stencil:
        Q.index_add_(0, at(p), q * W[0][p[0]] * W[1][p[1]] * W[2][p[2]])
    Qh = torch.fft.rfftn(Q.reshape(K))
    m, B = [], []
    Mn = _weights(torch.zeros(1, dtype=torch.float64))[0]
    for d in range(3):
        i = torch.arange(K[d] if d < 2 else K[d] // 2 + 1, dtype=torch.float64, device="cuda")
        b = sum(Mn[k + 1].item() * torch.exp(2j * math.pi * torch.remainder(i * k, K[d]) / K[d]) for k in range(ORDER - 1))
        shape = [1, 1, 1]
        shape[d] = -1
        B.append((1.0 / b.abs() ** 2).reshape(shape))
        m.append((torch.where(i > K[d] // 2, i - K[d], i) / L[d]).reshape(shape))
    mm = m[0] ** 2 + m[1] ** 2 + m[2] ** 2
    psi = torch.exp(-(math.pi / s.beta) ** 2 * mm) / mm * B[0] * B[1] * B[2] / (math.pi * V)
    psi[0, 0, 0] = 0.0
    twice = torch.full((K[2] // 2 + 1,), 2.0, dtype=torch.float64, device="cuda")
    twice[0] = twice[-1] = 1.0
    energy = 0.5 * (psi * Qh.abs() ** 2 * twice).sum()

    def back(h):
        h = torch.fft.ifftn(h, dim=(0, 1), norm="forward")
        return torch.fft.irfft(h, n=K[2], dim=2, norm="forward").reshape(-1)

    out = {"energy": energy}
    if method == "ik":
        G = [back(-2j * math.pi * m[d] * psi * Qh) for d in range(3)]
        F = [torch.zeros_like(q) for _ in range(3)]
        for p in stencil:
            w, a = W[0][p[0]] * W[1][p[1]] * W[2][p[2]], at(p)
            for d in range(3):
                F[d] += w * G[d][a]
        out["force"] = torch.stack([q * f for f in F], 1)
        return out
    phi = back(psi * Qh)
    dq = torch.zeros_like(q)
    g = [torch.zeros_like(q) for _ in range(3)]
    for p in stencil:
        v = phi[at(p)]
        w, e = [W[d][p[d]] for d in range(3)], [D[d][p[d]] for d in range(3)]
        dq += v * w[0] * w[1] * w[2]
        g[0] += v * e[0] * w[1] * w[2]
        g[1] += v * w[0] * e[1] * w[2]
        g[2] += v * w[0] * w[1] * e[2]
    dr = torch.stack([q * g[d] * (K[d] / L[d]) for d in range(3)], 1)
    out.update(dq=dq, dr=dr, force=-dr)
    return out


def _exact_grad(case, seed):
    s = _grad_system(case, seed)
    o = _spme(s, _cuda(s.charge), _cuda(s.pos), None)
    return {k: o[k].cpu() for k in ("energy", "dq", "dr")}


def _exact_hermite(case, seed):
    s = _of(case, seed)
    K, L, V, n = s.mesh, s.box, float(np.prod(s.box)), s.n
    st = _prepare_hermite(case, seed)
    half, nbin = case["half"], case["nbin"]
    CC, h = float(half), float(half) / nbin
    mv = torch.meshgrid(*[torch.fft.fftfreq(K[d], 1.0 / K[d], dtype=torch.float64, device="cuda") / L[d] for d in range(3)],
                        indexing="ij")
    mm = mv[0] ** 2 + mv[1] ** 2 + mv[2] ** 2
    mm[0, 0, 0] = 1.0
    base = torch.exp(-(math.pi / s.beta) ** 2 * mm) / (math.pi * V * mm)
    base[0, 0, 0] = 0.0
    mk = []
    for d in range(3):
        k = 2.0 * math.pi * mv[d].clone()
        if K[d] % 2 == 0:
            k.select(d, K[d] // 2).zero_()
        mk.append(k)

    def phi(c, u):
        one, zero = c.new_ones(1), c.new_zeros(1)
        v, e = torch.cat([one, c[:nbin]]), torch.cat([zero, c[nbin:]])
        a = u.abs()
        j = (a / h).detach().floor().long().clamp(max=nbin - 1)
        t = a / h - j
        p = (1 + 2 * t) * (1 - t) ** 2 * v[j] + t * (1 - t) ** 2 * h * e[j] + t * t * (3 - 2 * t) * v[j + 1] + \
            t * t * (t - 1) * h * e[j + 1]
        return torch.where(a < CC, p, torch.zeros_like(p))

    def forward(q, r, c):
        idx, W, b2 = [], [], 1.0
        for d in range(3):
            u = K[d] * torch.remainder(r[:, d] / L[d], 1.0)
            k0 = torch.floor(u.detach()).long() - half + 1
            k = k0[:, None] + torch.arange(2 * half, device="cuda")
            W.append(phi(c, u[:, None] - k))
            idx.append(torch.remainder(k, K[d]))
            i = torch.arange(-half, half + 1, dtype=torch.float64, device="cuda")
            m = torch.arange(K[d], dtype=torch.float64, device="cuda")
            b = (phi(c, i)[None, :] * torch.cos(2.0 * math.pi * torch.remainder(m[:, None] * i, K[d]) / K[d])).sum(1)
            shape = [1, 1, 1]
            shape[d] = -1
            b2 = b2 * b.reshape(shape) ** 2
        at = ((idx[0][:, :, None, None] * K[1] + idx[1][:, None, :, None]) * K[2] + idx[2][:, None, None, :]).reshape(-1)
        w = (W[0][:, :, None, None] * W[1][:, None, :, None] * W[2][:, None, None, :]).reshape(n, -1)
        Q = torch.zeros(K[0] * K[1] * K[2], dtype=torch.float64, device="cuda")
        Q = Q.index_add(0, at, (q[:, None] * w).reshape(-1))
        Qh, G = torch.fft.fftn(Q.reshape(K)), base / b2
        E = 0.5 * (G * (Qh.real ** 2 + Qh.imag ** 2)).sum()
        F = []
        for d in range(3):
            f = torch.fft.ifftn(1j * mk[d] * G * Qh, norm="forward").real.reshape(-1)
            F.append(-q * (w * f[at].reshape(n, -1)).sum(1))
        return E, torch.stack(F, 1)

    a = {k: [] for k in ("energy", "forces", "dE_dq", "dE_dr", "dE_dc")}
    b = {k: [] for k in ("loss", "dL_dq", "dL_dr", "dL_dc")}
    for cand in st["c"]:
        v = [t.detach().clone().requires_grad_(True) for t in (st["q"], st["r"], cand)]
        E, F = forward(*v)
        loss = ((F - st["fref"]) ** 2).sum() / n
        gE = torch.autograd.grad(E, v, retain_graph=True)
        gL = torch.autograd.grad(loss, v)
        for k, t in zip(a, (E, F) + gE):
            a[k].append(t.detach().cpu())
        for k, t in zip(b, (loss,) + gL):
            b[k].append(t.detach().cpu())
    return [{k: torch.stack(t) for k, t in o.items()} for o in (a, b)]


def _exact_errmap(case, seed):
    s = _of(case, seed)
    K, L, V, n = (case["k0"], case["k1"], case["k2"]), s.box, float(np.prod(s.box)), case["order"]
    N = math.prod(K)
    ii = [torch.arange(k, device="cuda") for k in K]
    cen = [torch.where(i > k // 2, i - k, i).double() for i, k in zip(ii, K)]

    def along(v, d):
        shape = [1, 1, 1]
        shape[d] = -1
        return v.reshape(shape)

    m = [along(cen[d] / L[d], d) for d in range(3)]
    mm = m[0] ** 2 + m[1] ** 2 + m[2] ** 2
    mm[0, 0, 0] = 1.0
    fm = torch.exp(-(math.pi / s.beta) ** 2 * mm) / mm / (2.0 * math.pi * V)
    fm[0, 0, 0] = 0.0
    g = []
    for d in range(3):
        v = -4.0 * math.pi * fm * m[d]
        if K[d] % 2 == 0:
            v.select(d, K[d] // 2).zero_()
        g.append(v)
    u = [2.0 * math.pi * cen[d] / K[d] for d in range(3)]

    def alias(d, k):
        # (u + 2 pi k)^-n over its sum for |l| <= 3, multiplied through by u^n (finite at u = 0)
        ratio = sum((u[d] / (u[d] + 2.0 * math.pi * l)) ** n for l in range(-3, 4) if l)
        return (u[d] / (u[d] + 2.0 * math.pi * k)) ** n / (1.0 + ratio)

    ift = lambda v: torch.fft.ifftn(1j * v, norm="forward")  # noqa: E731
    k2b, tot = torch.zeros(K, dtype=torch.float64, device="cuda"), torch.zeros(K, dtype=torch.float64, device="cuda")
    for k in range(-4, 5):
        if k:
            for d in range(3):
                a = along(alias(d, k), d)
                tot = tot + 2.0 * a
                k2b = k2b + sum(ift(v * a).abs() ** 2 for v in g) * (V / N)
    k2a = torch.fft.fftn(sum(ift(v * tot).abs() ** 2 for v in g) * (V / N) + 2.0 * k2b + 0j)
    ix = [np.minimum((s.pos[:, d] / (L[d] / K[d])).astype(np.int64), K[d] - 1) for d in range(3)]
    at = ((ix[0] * K[1] + ix[1]) * K[2] + ix[2])[s.charge != 0]
    rho = [_cuda(np.bincount(at, weights=w, minlength=N).reshape(K)) * (N / V)
           for w in (s.charge[s.charge != 0], np.ones(at.size))]
    r1, r2 = [torch.fft.fftn(r) * (V / N) for r in rho]
    e = (torch.fft.ifftn(k2a * r2, norm="forward") / V).real
    for v in g:
        e = e + (torch.fft.ifftn(1j * v * tot * V * r1, norm="forward") / V).real ** 2
    return e.sqrt().cpu().numpy()


def _exact_ikerr(case, seed):
    K, L, beta, nbin, cut, CC = case["k"], 30.0, 0.95, case["nbin"], 10, 2.0
    M, h, kmax = K * int(400.0 * (nbin / CC)), CC / nbin, K // 2 + 10 * K
    x = torch.arange(M, dtype=torch.float64, device="cuda") * (K / M)
    x = torch.where(x > K / 2, x - K, x).abs()
    hats = []
    for slope in (False, True):
        for j in range(nbin + 1):
            t = x / h - j
            lo, up = t + 1.0, t
            v = torch.where(t < 0, lo * lo * (lo - 1) * h if slope else lo * lo * (3 - 2 * lo),
                            up * (1 - up) ** 2 * h if slope else (1 + 2 * up) * (1 - up) ** 2)
            v = torch.where((t.abs() < 1) & (x <= CC), v, 0.0)
            hats.append((torch.fft.fft(v + 0j) / M).real[:kmax + 1])
    hat0, hb = hats[0], torch.stack(hats[1:nbin + 1] + hats[nbin + 2:])
    i = torch.arange(-(K // 2), K // 2 + 1, device="cuda")
    m = i.double() / L
    mm = (m[:, None, None] ** 2 + m[None, :, None] ** 2 + m[None, None, :] ** 2)
    w = 32.0 * math.pi ** 2 * torch.exp(-2.0 * (math.pi / beta) ** 2 * mm) / torch.where(mm > 0, mm, 1.0)
    w = torch.where(mm > 0, w, 0.0).sum((1, 2))
    c = _candidates(case["cand"], 2, nbin, seed).requires_grad_(True)
    phi = hat0 + c @ hb
    T = sum(phi[:, (i + l * K).abs()] ** 2 for l in range(-cut, cut + 1) if l) / phi[:, i.abs()] ** 2
    s = 3.0 * (w * T).sum(1) / (2.0 * math.pi * L ** 3) ** 2
    loss = torch.sqrt(s * 20736.0) * 138.93545756169981341199
    grad, = torch.autograd.grad(loss.sum(), c)
    return {"loss": loss.detach().cpu(), "grad": grad.cpu()}


def _exact_ewald(case, seed):
    s = _of(case, seed)
    x, q, V = _cuda(s.pos), _cuda(s.charge), float(np.prod(s.box))
    M = case["k"] // 2
    i = torch.arange(-M, M + 1, dtype=torch.float64, device="cuda")
    m = torch.stack(torch.meshgrid(i, i, i, indexing="ij"), -1).reshape(-1, 3) / _cuda(s.box)
    m = m[m.abs().sum(1) > 0]
    F, E = torch.zeros_like(x), 0.0
    for mc in m.split(8192):
        ph = 2.0 * math.pi * torch.remainder(mc @ x.T, 1.0)
        cs, sn = torch.cos(ph), torch.sin(ph)
        sr, si = cs @ q, sn @ q
        mm = (mc ** 2).sum(1)
        ex = torch.exp(-(math.pi / s.beta) ** 2 * mm) / mm
        E = E + (ex * (sr ** 2 + si ** 2)).sum() / (2.0 * math.pi * V)
        co = (sr[:, None] * sn - si[:, None] * cs) * (2.0 / V * ex)[:, None]
        F = F + q[:, None] * (co.T @ mc)
    return {"energy": float(E), "forces": F.cpu().numpy()}
