"""The measured workloads of the B200 Kohn-Sham solver: what a program built on it has it do.

Three families, each called the way a user's program calls it:

- ``hpsi``: H psi on device fields (``ks_b200.hpsi_device``), the operator a caller with its own eigensolver or
  propagator applies to a block of orbitals;
- ``gram``: the subspace products S^T [S | T] on device fields (``ks_b200.gram_device_noalloc``);
- whole solves through ``ks_b200.GpuSolver`` and the drivers above it: a cold SCF with forces, energies and the density
  image (``scf``), a cold solve followed by warm velocity-Verlet steps (``md``), and a batch of independent molecules
  (``batch``).

Sizes and settings are the workloads of this repository's configurations, tests and benchmark. Geometries carry a
seeded Gaussian jitter, so that another seed is another molecule.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "atomic-sandbox_b200"))
import ks_b200 as ks  # noqa: E402
import ks_drivers as drv  # noqa: E402

MOLECULES = {
    # name: (geometry, electrons up, electrons down)
    "H2": (drv.h2, 1, 1),
    "LiH": (drv.lih, 2, 2),
    "H2O": (drv.h2o, 5, 5),
    "NH3": (drv.nh3, 5, 5),
    "CH4": (drv.ch4, 5, 5),
    "HF": (drv.hf, 5, 5),
    "C4H10": (drv.butane_anti, 17, 17),
}
COEFF = (-205.0 / 72.0, 8.0 / 5.0, -1.0 / 5.0, 8.0 / 315.0, -1.0 / 560.0)  # 8th-order second difference


def _scf(name, molecule, n, h, sigma, mixed, **more):
    case = {"name": name, "kind": "scf", "molecule": molecule, "n": n, "h": h, "sigma": sigma, "mixed": mixed, "extra": 3,
            "jitter": 0.05, "fermi_dirac": False, "pseudo": False, "tol": 1e-6}
    case.update(more)
    return case


def listed():
    return [
        # the smallest operator call: a few orbitals of a small molecule's box, where the launch counts
        {"name": "hpsi_3x33", "kind": "hpsi", "n": 33, "count": 3, "h": 0.25},
        # the [W | P] block of the water solve, in and out of the L2
        {"name": "hpsi_16x95", "kind": "hpsi", "n": 95, "count": 16, "h": 0.25},
        # a butane-sized block of 2 x 20 orbitals, from HBM
        {"name": "hpsi_40x128", "kind": "hpsi", "n": 128, "count": 40, "h": 0.2},
        # the subspace products of an 8-band LOBPCG step
        {"name": "gram_24_24x95", "kind": "gram", "n": 95, "m": 24, "mt": 24},
        # a small cold solve: many short launches and readbacks
        _scf("h2_48_plain", "H2", 48, 0.25, 0.5, False),
        # the benchmark molecule, in both forms of the subspace products
        _scf("h2o_95_plain", "H2O", 95, 0.25, 0.5, False),
        _scf("h2o_95_mixed", "H2O", 95, 0.25, 0.5, True),
        # the largest solve: 20 bands per spin on 128^3 (the density floor of 34 electrons asks for 2e-6)
        _scf("c4h10_128_mixed", "C4H10", 128, 0.2, 0.5, True, jitter=0.02, tol=2e-6),
        # molecular dynamics: a cold solve, then warm solves of moved nuclei with forces
        {"name": "nh3_md_64_mixed", "kind": "md", "molecule": "NH3", "n": 64, "h": 0.25, "sigma": 0.25, "mixed": True, "extra": 3,
         "jitter": 0.05, "steps": 3, "tol": 1e-6},
        # Fermi-Dirac occupations at the provider's temperature, an odd grid
        _scf("lih_fd_49", "LiH", 49, 0.25, 0.25, False, extra=4, fermi_dirac=True),
        # a pseudised centre: the nonlocal operator in every H psi and the partial core in XC
        _scf("h2o_pseudo_65", "H2O", 65, 0.25, 0.5, True, pseudo=True),
        # a batch of molecules on grids of their own, solved concurrently
        {"name": "batch_6", "kind": "batch", "jobs": "H2:48 H2O:57 NH3:53 CH4:64 LiH:51 HF:60", "mixed": True, "workers": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("hpsi", "hpsi", "gram", "scf", "scf", "fd", "pseudo", "md", "batch"))
    if kind == "hpsi":
        n = _log_int(rng, 33, 128)
        # at most the points of the largest listed block
        return {"kind": "hpsi", "n": n, "count": _log_int(rng, 1, min(64, 40 * 128 ** 3 // n ** 3)), "h": round(rng.uniform(0.18, 0.3), 3)}
    if kind == "gram":
        n = _log_int(rng, 33, 95)
        m = rng.randint(2, 24)
        return {"kind": "gram", "n": n, "m": m, "mt": rng.choice((m, m, rng.randint(1, 24)))}
    h = round(rng.uniform(0.22, 0.28), 3)
    if kind == "scf":
        name = rng.choice(("H2", "LiH", "H2O", "NH3", "CH4", "HF"))
        case = _scf("", name, rng.randint(48, 96), h, 0.5, rng.random() < 0.5)
    elif kind == "fd":
        case = _scf("", "LiH", rng.randint(41, 56), h, round(h, 3), rng.random() < 0.5, extra=4, fermi_dirac=True)
    elif kind == "pseudo":
        case = _scf("", "H2O", rng.randint(48, 80), h, 0.5, rng.random() < 0.5, pseudo=True)
    elif kind == "md":
        return {"kind": "md", "molecule": rng.choice(("H2O", "NH3", "CH4")), "n": rng.randint(48, 72), "h": h, "sigma": h,
                "mixed": rng.random() < 0.5, "extra": 3, "jitter": 0.05, "steps": rng.randint(2, 4), "tol": 1e-6}
    else:
        jobs = " ".join("%s:%d" % (rng.choice(("H2", "LiH", "H2O", "NH3", "CH4", "HF")), rng.randint(48, 64)) for _ in range(rng.randint(3, 8)))
        return {"kind": "batch", "jobs": jobs, "mixed": rng.random() < 0.5, "workers": rng.choice((2, 4, 8))}
    case.pop("name")
    return case


# ---- device fields: element (i, j, k) at (k n + j) P + i, pad columns 0
def _axes(n, h, dtype):
    c = (torch.arange(n, device="cuda", dtype=dtype) - (n - 1) / 2) * h
    return c.view(1, 1, n), c.view(1, n, 1), c.view(n, 1, 1)


def _orbitals(n, h, count, g, out):
    """Smooth localised orbitals (Gaussians times a linear form) with, on every second one, a rough part as the
    search directions of an eigensolver have."""
    x, y, z = _axes(n, h, torch.float64)
    par = torch.rand(count, 8, generator=g, dtype=torch.float64) * 2 - 1
    for v in range(count):
        p = par[v].tolist()
        r2 = (x - p[0]) ** 2 + (y - p[1]) ** 2 + (z - p[2]) ** 2
        f = (p[3] + p[4] * x + p[5] * y + p[6] * z) * torch.exp(-(0.6 + 0.4 * p[7]) * r2)
        if v % 2:
            f = f + 1e-3 * (torch.rand(n, n, n, device="cuda", dtype=torch.float64, generator=torch.Generator("cuda").manual_seed(
                int(torch.randint(1 << 30, (1,), generator=g)))) - 0.5)
        out[v, :, :, :n] = f.float()


def _block(n, count):
    return torch.zeros(count, n, n, ks.field_pitch(n), device="cuda")


def _oxygen(h):
    """An analytic six-valence-electron ion: Gaussians times the compact bump (1 - (d/rc)^2)^3, with a short-range core,
    a partial core and one s and one p projector."""
    du = h / 256

    def table(amp, width, rc):
        d = np.arange(int(math.ceil(rc / du)) + 4) * du
        return np.where(d < rc, amp * np.exp(-d * d / (2 * width * width)) * (1 - np.clip(d / rc, 0, 1) ** 2) ** 3, 0.0)
    return ks.Species(z=8, z_v=6.0, sigma_lr=2 * h, du=du, v_sr=table(3.0, 0.35, 1.5), r_sr=1.5, rho_pc=table(0.8, 0.30, 1.2), pc_radius=1.2,
                      projectors=[ks.Projector(0, 1.2, 1.6, table(1.5, 0.40, 1.6)), ks.Projector(1, -0.6, 1.6, table(2.0, 0.45, 1.6))])


def _nuclei(molecule, jitter, seed):
    return drv.jittered(MOLECULES[molecule][0](), jitter, seed)


def _jobs(case):
    return [(j.split(":")[0], int(j.split(":")[1])) for j in case["jobs"].split()]


def prepare(case, seed):
    kind = case["kind"]
    g = torch.Generator().manual_seed(seed)
    if kind == "hpsi":
        n, count, h = case["n"], case["count"], case["h"]
        psi, v = _block(n, count), _block(n, 1)
        _orbitals(n, h, count, g, psi)
        x, y, z = _axes(n, h, torch.float64)
        c = torch.rand(3, generator=g, dtype=torch.float64).tolist()
        r = torch.sqrt((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2).clamp_min(1e-6)
        v[0, :, :, :n] = (-8.0 * torch.erf(r / (0.5 * math.sqrt(2.0))) / r + 6.0 / (1.0 + r)).float()
        return {"case": case, "psi": psi, "v": v, "out": torch.empty_like(psi)}
    if kind == "gram":
        n, m, mt = case["n"], case["m"], case["mt"]
        s, t = _block(n, m), _block(n, mt)
        _orbitals(n, 0.25, m, g, s)
        _orbitals(n, 0.25, mt, g, t)
        return {"case": case, "s": s, "t": t, "out": torch.empty(m, m + mt, device="cuda", dtype=torch.float64)}
    if kind == "batch":
        jobs = []
        for i, (name, n) in enumerate(_jobs(case)):
            jobs.append({"nuclei": _nuclei(name, 0.05, seed + i), "n": n, "h": 0.25, "n_up": MOLECULES[name][1], "n_dn": MOLECULES[name][2],
                         "settings": ks.ScfSettings(sigma=0.5)})
        return {"case": case, "jobs": jobs}
    # the solver a program keeps for its grid, and where it wants the density image
    solver = ks.GpuSolver(case["n"], case["h"], gram_mode=1 if case["mixed"] else 0, n_extra=case["extra"], init_mode=1)
    state = {"case": case, "solver": solver, "nuclei": _nuclei(case["molecule"], case["jitter"], seed),
             "volume": torch.empty(case["n"], case["n"], case["n"], device="cuda")}
    if kind == "md":
        state["settings"] = ks.ScfSettings(sigma=case["sigma"], tol=case["tol"])
        return state
    up, dn = MOLECULES[case["molecule"]][1:]
    if case["pseudo"]:  # the 1s pair is in the ion's core
        solver.set_ionic([_oxygen(case["h"])])
        up, dn = up - 1, dn - 1
    state["system"] = ks.System(state["nuclei"], up, dn)
    state["settings"] = ks.ScfSettings(sigma=case["sigma"], tol=case["tol"], occupations="fermi_dirac" if case["fermi_dirac"] else "aufbau")
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "hpsi":
        ks.hpsi_device(torch.cuda.current_stream().cuda_stream, case["n"], case["h"], case["count"], state["psi"].data_ptr(),
                       state["v"].data_ptr(), state["out"].data_ptr())
        return state["out"]
    if kind == "gram":
        ks.gram_device_noalloc(torch.cuda.current_stream().cuda_stream, case["n"], case["m"], state["s"].data_ptr(), case["mt"],
                               state["t"].data_ptr(), state["out"].data_ptr())
        return state["out"]
    if kind == "batch":
        out = ks.solve_batch(state["jobs"], workers=case["workers"], gram_mode=1 if case["mixed"] else 0)
        bad = [r["error"] for r in out if r["status"] != ks.KS_OK]
        if bad:
            raise ks.QmError(bad[0])
        return {"energy": np.array([r["stats"]["energy"]["total"] for r in out]), "forces": np.concatenate([r["forces"] for r in out])}
    solver, volume = state["solver"], state["volume"]
    if kind == "md":
        _, up, dn = MOLECULES[case["molecule"]]
        traj = drv.velocity_verlet(solver, state["nuclei"], up, dn, state["settings"], 0.5 / drv.FS_PER_AU, case["steps"])
        solver.copy_density_to_volume(volume.data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"energy": np.array([t["potential"] for t in traj]), "velocities": traj[-1]["velocities"], "density": volume}
    stats = solver.solve(state["system"], state["settings"])
    solver.copy_density_to_volume(volume.data_ptr(), torch.cuda.current_stream().cuda_stream)
    forces = solver.forces(state["nuclei"], case["sigma"])
    n_up, n_dn = state["system"].n_up, state["system"].n_dn
    levels = [e[:c] for e, c in zip(solver.evals(), (n_up, n_dn))]
    return {"energy": stats["energy"]["total"], "levels": np.concatenate(levels), "forces": forces, "density": volume}


def _solve_work(n, bands, iterations):
    """The passes of the eigensolver's iterations over both spins' blocks: five H applies per vector (three
    preconditioner sweeps, H W and H P, H X), the products S^T [S | H S] of S = [X W P] and the update of X and P; X, W, P
    and V read and X, P written once per iteration."""
    pts = n ** 3
    m = 3 * bands
    return {"bytes": iterations * pts * 4.0 * (m + 1 + 2 * bands),
            "flops": iterations * pts * (6.0 * bands * 75 + 2.0 * m * (m + 1) + 2.0 * m * 2 * bands)}


def work(case):
    kind = case["kind"]
    if kind == "hpsi":
        pts = case["n"] ** 3
        return {"bytes": (8.0 * case["count"] + 4.0) * pts, "flops": 75.0 * case["count"] * pts}
    if kind == "gram":
        m, mt, pts = case["m"], case["mt"], case["n"] ** 3
        return {"bytes": 4.0 * (m + mt) * pts, "flops": (m * (m + 1.0) + 2.0 * m * mt) * pts}
    # nominal counts: about 16 SCF steps of 16 iterations per spin for a cold solve, a third of that for a warm one
    if kind == "batch":
        each = [_solve_work(n, MOLECULES[name][1] + 3, 512) for name, n in _jobs(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    up, dn = MOLECULES[case["molecule"]][1:]
    bands = (up + dn) / 2 + case["extra"]
    return _solve_work(case["n"], bands, 512 * (1 + (case["steps"] / 3 if kind == "md" else 0)))


def tolerance(case):
    kind = case["kind"]
    if kind == "hpsi":  # measured against exact(): up to 5.5e-8, largest where the two terms cancel near a nucleus
        return {"rel": 5e-7, "max": 2e-5}
    if kind == "gram":  # measured against exact(): up to 1.1e-7
        return {"rel": 5e-7, "max": 5e-6}
    # two solves of one molecule from other starting orbitals or with the other form of the products, both converged to
    # the same tolerance: up to 1.3e-5 in the forces, 5e-6 in the density and the levels
    return {"rel": 1e-4, "max": 1e-3}


def exact(case, seed):
    """64-bit answers of the operator and of the products. A whole solve has none: a 64-bit SCF takes minutes."""
    kind = case["kind"]
    if kind not in ("hpsi", "gram"):
        return None
    state = prepare(case, seed)
    if kind == "gram":
        s = state["s"].double().flatten(1)
        return s @ torch.cat([s, state["t"].double().flatten(1)]).T
    n, h = case["n"], case["h"]
    v = state["v"][0, :, :, :n].double()
    out = torch.zeros(state["psi"].shape, device="cuda", dtype=torch.float64)
    for i in range(case["count"]):
        f = state["psi"][i, :, :, :n].double()
        pad = torch.nn.functional.pad(f, (4,) * 6)
        lap = 3 * COEFF[0] * f
        for axis in range(3):
            for m in range(1, 5):
                for s in (-m, m):
                    at = [slice(4, 4 + n)] * 3
                    at[axis] = slice(4 + s, 4 + s + n)
                    lap = lap + COEFF[m] * pad[tuple(at)]
        out[i, :, :, :n] = -0.5 / (h * h) * lap + v * f
    return out
