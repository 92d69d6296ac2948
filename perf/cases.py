"""Measured cases: what a user of this framework has it do, through its public
entry points, over the range of sizes, precisions and options it takes.

Three kinds of case:

``march``
    A run of a meshed box: materials and boundaries are in hand as an engine
    (``FitProblem.build_engine``), one pass advances it by ``steps`` leapfrog
    steps in the marching loop (``FitRun``, with its stored-energy checks) and
    reads back what the solver hands its caller: the fields, the recorded port
    voltages and currents, and the monitors' running-DFT bins.  ``stencil`` is
    ``"default"`` (a handle as it is created, which is what the drop-in solver
    marches on) or ``"slab"`` (the form the serving loop and the benchmark
    select).
``dispersive``
    The same for the dispersive-slab box with its TF/SF plane wave.
``serve``
    Whole S-parameter requests through the serving loop: port modes, device
    setup, all excitations, S-matrices.
``modes``
    The sparse port-mode eigensolve that every waveguide-port setup calls.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from magnelio_b200.engine import sparse_eigs
from magnelio_b200.problem import CpmlFace, DftMonitor, FitProblem, LumpedPort, MaterialSetup
from magnelio_b200.runloop import FitRun
from magnelio_b200.serving import Request, ServingLoop
from magnelio_b200.workloads import dispersive_slab, waveguide_section_modal

C0 = 299792458.0
MU0 = 1.25663706212e-6  # CODATA 2018
EPS0 = 1.0 / (MU0 * C0 * C0)
R_PORT = 50.0
E_COMPONENTS = ("Ex", "Ey", "Ez")


def _march(name, nx, ny, nz, steps, *, batch=1, precision="single", coef="native", stencil="default", faces="xyz",
           layers=8, planes=0, n_freq=16, lossy=False):
    return {"name": name, "kind": "march", "nx": nx, "ny": ny, "nz": nz, "steps": steps, "batch": batch,
            "precision": precision, "coef": coef, "stencil": stencil, "faces": faces, "layers": layers,
            "planes": planes, "n_freq": n_freq, "lossy": lossy}


def listed():
    return [
        # a coarse waveguide section, the smallest mesh in use: every step is launches and latency
        _march("guide_small", 23, 11, 41, 500, faces="z"),
        # the ordinary antenna / connector box of the drop-in solver: CPML all round, three DFT planes
        _march("box_mid", 97, 104, 89, 500, planes=3),
        # a large ragged box in the drop-in solver
        _march("box_large_ragged", 251, 187, 233, 500, planes=1),
        # the headline box of the benchmark (256^3, ten layers, three planes), in the form it selects
        _march("box_256_slab", 256, 256, 256, 800, stencil="slab", layers=10, planes=3),
        # the largest mesh: a simulation of 49 M cells
        _march("box_largest_slab", 400, 384, 320, 400, stencil="slab", layers=10),
        # four excitations of one mesh as one batch
        _march("batch4_mid", 95, 88, 110, 400, batch=4),
        # a served waveguide request: eight channels, 16-bit coefficients, PEC walls
        _march("batch8_guide_f16", 72, 32, 127, 600, batch=8, coef="f16", faces="z"),
        # a double-precision run (convergence studies)
        _march("double_mid", 81, 75, 90, 400, precision="double", planes=1),
        # lossy dielectrics: every update coefficient differs from one
        _march("lossy_mid_slab", 129, 118, 140, 500, stencil="slab", planes=1, lossy=True),
        # a frequency-dependent material under a plane wave: ADE states, TF/SF faces
        {"name": "dispersive_mid", "kind": "dispersive", "nx": 90, "ny": 84, "nz": 120, "steps": 400,
         "stencil": "default", "n_freq": 16},
        # the serving loop on small waveguide requests, from the mesh to the S-matrix
        {"name": "serve_small", "kind": "serve", "requests": 3, "cells_lo": 20**3, "cells_hi": 40**3, "steps": 1200,
         "modes_in": 2, "modes_out": 1, "lumped": 1, "ridged": False, "n_freq": 51},
        # the port modes of a fine waveguide plane
        {"name": "port_modes", "kind": "modes", "nu": 104, "nv": 46, "n_modes": 3},
    ]


def draw(rng):
    kind = rng.choice(["march"] * 6 + ["dispersive", "serve", "modes"])
    if kind == "modes":
        return {"kind": "modes", "nu": rng.randint(30, 160), "nv": rng.randint(16, 70), "n_modes": rng.randint(1, 4)}
    if kind == "serve":
        lo = int(round(math.exp(rng.uniform(math.log(16.0), math.log(30.0))))) ** 3
        return {"kind": "serve", "requests": rng.randint(1, 3), "cells_lo": lo,
                "cells_hi": int(lo * rng.uniform(1.1, 3.0)), "steps": rng.randint(600, 1500),
                "modes_in": rng.randint(1, 2), "modes_out": rng.randint(1, 2), "lumped": rng.randint(0, 2),
                "ridged": rng.random() < 0.5, "n_freq": rng.randint(21, 101)}
    if kind == "dispersive":
        return {"kind": "dispersive", "nx": rng.randint(40, 110), "ny": rng.randint(40, 110), "nz": rng.randint(60, 130),
                "steps": rng.randint(100, 400), "stencil": rng.choice(["default", "slab"]), "n_freq": rng.randint(4, 32)}
    cells = math.exp(rng.uniform(math.log(1.0e4), math.log(1.5e7)))
    ra, rb = math.exp(rng.uniform(-0.5, 0.5)), math.exp(rng.uniform(-0.5, 0.5))
    s = (cells / (ra * rb)) ** (1.0 / 3.0)
    nx, ny, nz = max(9, int(s * ra)), max(9, int(s * rb)), max(40, int(s))
    cells = nx * ny * nz
    batch = rng.choice([1, 1, 1, 2, 4, 8]) if cells < 2.0e6 else 1
    precision = "double" if batch == 1 and cells < 4.0e6 and rng.random() < 0.2 else "single"
    coef = "f16" if precision == "single" and rng.random() < 0.15 else "native"
    layers = rng.choice([0, 6, 8, 10])
    layers = min(layers, (min(nx, ny, nz) - 2) // 2)
    return {"kind": "march", "nx": nx, "ny": ny, "nz": nz,
            "steps": max(50, min(600, int(2.5e9 / (cells * batch)))), "batch": batch, "precision": precision,
            "coef": coef, "stencil": rng.choice(["default", "slab"]), "faces": rng.choice(["xyz", "xyz", "z"]),
            "layers": layers, "planes": rng.choice([0, 1, 3]) if batch == 1 else 0, "n_freq": rng.randint(4, 32),
            "lossy": rng.random() < 0.25 and cells < 4.0e6}


# ---------------------------------------------------------------------------
# The meshed box: grid, materials, absorber tables, ports (plain numpy)
# ---------------------------------------------------------------------------
def _dual(d):
    return np.concatenate([d[:1], 0.5 * (d[:-1] + d[1:]), d[-1:]])


def _shapes(nx, ny, nz):
    return {"Ex": (nx, ny + 1, nz + 1), "Ey": (nx + 1, ny, nz + 1), "Ez": (nx + 1, ny + 1, nz),
            "Hx": (nx + 1, ny, nz), "Hy": (nx, ny + 1, nz), "Hz": (nx, ny, nz + 1)}


def _flat(shapes, comp, index):
    """Flat indices into the E vector of the sub-box ``index`` (three slices) of component ``comp``."""
    off = sum(int(np.prod(shapes[c])) for c in E_COMPONENTS[:E_COMPONENTS.index(comp)])
    axes = [np.arange(n)[s] for n, s in zip(shapes[comp], index)]
    return (off + np.ravel_multi_index(np.ix_(*axes), shapes[comp]).ravel()).astype(np.int64)


def _cpml(d, side, layers, dt):
    """Graded CFS-PML recursion tables (b, c, 1 - 1/kappa) of one face."""
    w = d[:layers] if side == "min" else d[-layers:][::-1]  # outermost layer first
    depth = w.sum()
    rho = 1.0 - (np.cumsum(w) - 0.5 * w) / depth
    sigma = 4.0 * EPS0 * C0 * math.log(1e8) / (2.0 * depth) * rho**3
    kappa, alpha = 1.0 + 6.0 * rho**3, 0.02 * (1.0 - rho)
    b = np.exp(-(sigma / kappa + alpha) * dt / EPS0)
    c = sigma / (kappa * sigma + kappa**2 * alpha) * (1.0 - b)
    ck = 1.0 - 1.0 / kappa
    return tuple(t if side == "min" else t[::-1].copy() for t in (b, c, ck))


class _Box:
    """What a mesher hands the solver for one march case: graded grid, brick
    materials with conformal averages on the brick surfaces, PEC walls or
    CPML, one gap port per field set, DFT planes."""

    def __init__(self, case, seed):
        rng = np.random.default_rng(seed)
        n = (case["nx"], case["ny"], case["nz"])
        self.n, self.batch, self.steps = n, case["batch"], case["steps"]
        self.shapes = _shapes(*n)
        self.d = [1e-3 * rng.uniform(0.8, 1.2, v) for v in n]
        self.dt = 0.95 / (C0 * math.sqrt(sum(1.0 / v.min() ** 2 for v in self.d)))
        n_bricks = 16
        self.eps_r = np.concatenate([[1.0], rng.uniform(1.0, 10.0, n_bricks)])
        self.sigma = np.concatenate([[1e-3], rng.uniform(0.01, 0.5, n_bricks)]) if case["lossy"] else None
        self.mat_id = np.zeros(n, np.int32)
        cat1 = []
        for q in range(n_bricks):
            size = [max(1, int(v * rng.uniform(0.05, 0.3))) for v in n]
            lo = [int(rng.integers(0, v - s + 1)) for v, s in zip(n, size)]
            sl = [slice(a, a + s) for a, s in zip(lo, size)]
            self.mat_id[tuple(sl)] = q + 1
            for axis in range(3):  # the surface edges of the brick's two faces on this axis
                for plane in (sl[axis].start, sl[axis].stop):
                    for comp in range(3):
                        if comp == axis:
                            continue
                        idx = list(sl)
                        idx[axis] = slice(plane, plane + 1)
                        cat1.append(_flat(self.shapes, E_COMPONENTS[comp], idx))
        self.cat1 = np.unique(np.concatenate(cat1))
        self.cat1_eps = rng.uniform(1.0, 6.0, self.cat1.size)
        self.cpml = []
        if case["layers"]:
            for face in ("xmin", "xmax", "ymin", "ymax", "zmin", "zmax"):
                if face[0] in case["faces"]:
                    axis = "xyz".index(face[0])
                    self.cpml.append((axis, face, *_cpml(self.d[axis], face[1:], case["layers"], self.dt)))
        self.pec = np.zeros(0, np.int64)
        if case["faces"] == "z":  # a guide: PEC side walls
            every = slice(None)
            walls = []
            for end in (0, -1):
                s = slice(0, 1) if end == 0 else slice(-1, None)
                walls += [_flat(self.shapes, c, (s, every, every)) for c in ("Ey", "Ez")]
                walls += [_flat(self.shapes, c, (every, s, every)) for c in ("Ex", "Ez")]
            self.pec = np.unique(np.concatenate(walls))
        # one y-directed gap port per field set along the middle of the box
        lo, hi = case["layers"] + 2, n[2] - case["layers"] - 2
        self.port = [(n[0] // 2, n[1] // 2, lo + (hi - lo) * (b + 1) // (self.batch + 1)) for b in range(self.batch)]
        t = (np.arange(4096) + 1) * self.dt
        f_max = rng.uniform(14e9, 20e9)
        width, mid = f_max - 2e9, 0.5 * (f_max + 2e9)
        x = (t - 4.0 / width) * math.pi * width / 2.0
        self.pulse = 2.0 * math.sqrt(R_PORT) * np.exp(-x * x) * np.cos(2.0 * math.pi * mid * (t - 4.0 / width))
        self.freqs = np.linspace(2e9, f_max, case["n_freq"])
        self.planes = []
        for axis in range(case["planes"]):
            box = [(0, v) for v in n]
            box[axis] = (n[axis] // 2, n[axis] // 2 + 1)
            self.planes.append(tuple(box))

    def coefficients(self, device):
        """alpha_E, beta_E, M_eps, beta_H, M_mu as float64 tensors per component."""
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=device)  # noqa: E731
        (dx, dy, dz), (ax, ay, az) = [t(v) for v in self.d], [t(_dual(v)) for v in self.d]
        X, Y, Z = (lambda v: v[:, None, None]), (lambda v: v[None, :, None]), (lambda v: v[None, None, :])
        geo_e = [Y(ay) * Z(az) / X(dx), X(ax) * Z(az) / Y(dy), X(ax) * Y(ay) / Z(dz)]
        geo_h = [Y(dy) * Z(dz) / X(ax), X(dx) * Z(dz) / Y(ay), X(dx) * Y(dy) / Z(az)]
        mat = torch.as_tensor(self.mat_id, device=device).long()
        last = [torch.clamp(torch.arange(v + 1, device=device), max=v - 1) for v in self.n]
        owner = [mat[:, last[1]][:, :, last[2]], mat[last[0]][:, :, last[2]], mat[last[0]][:, last[1]]]
        eps, sig = t(self.eps_r), None if self.sigma is None else t(self.sigma)
        cat1 = [torch.as_tensor(self.cat1, device=device), t(self.cat1_eps)]
        pec = torch.as_tensor(self.pec, device=device)
        a_e, b_e, m_e = [], [], []
        off = 0
        for g, own in zip(geo_e, owner):
            rel = eps[own].reshape(-1)
            here = (cat1[0] >= off) & (cat1[0] < off + rel.numel())
            rel[cat1[0][here] - off] = cat1[1][here]
            m = EPS0 * rel.view(own.shape) * g
            loss = 0.0 if sig is None else 0.5 * self.dt * sig[own] * g
            a, b = (m - loss) / (m + loss), self.dt / (m + loss)
            wall = pec[(pec >= off) & (pec < off + rel.numel())] - off
            a.view(-1)[wall] = 0.0
            b.view(-1)[wall] = 0.0
            a_e.append(a)
            b_e.append(b)
            m_e.append(m)
            off += rel.numel()
        m_h = [MU0 * g for g in geo_h]
        return a_e, b_e, m_e, [self.dt / m for m in m_h], m_h

    def port_mass(self, b):
        """M_eps and flat index of field set b's port edge (an Ey edge; a port
        on a brick surface keeps the conformal average)."""
        i, j, k = self.port[b]
        flat = int(_flat(self.shapes, "Ey", (slice(i, i + 1), slice(j, j + 1), slice(k, k + 1)))[0])
        at = np.searchsorted(self.cat1, flat)
        eps = (self.cat1_eps[at] if at < self.cat1.size and self.cat1[at] == flat
               else self.eps_r[self.mat_id[min(i, self.n[0] - 1), j, min(k, self.n[2] - 1)]])
        g = _dual(self.d[0])[i] * _dual(self.d[2])[k] / self.d[1][j]
        sig = 0.0 if self.sigma is None else 0.5 * self.dt * g * self.sigma[
            self.mat_id[min(i, self.n[0] - 1), j, min(k, self.n[2] - 1)]]
        return EPS0 * eps * g + sig, flat

    def problem(self):
        nx, ny, nz = self.n
        grid = dict(nx=nx, ny=ny, nz=nz, dt=self.dt, dx=self.d[0], dy=self.d[1], dz=self.d[2], batch=self.batch)
        if self.sigma is None:
            prob = FitProblem(**grid, alpha_E=None, beta_E=None, alpha_H=None, beta_H=None,
                              materials=MaterialSetup(self.mat_id, self.eps_r, self.cat1, self.cat1_eps, self.pec))
        else:  # conductive materials: the solver's host arrays
            a_e, b_e, m_e, b_h, m_h = (torch.cat([v.reshape(-1) for v in c]).cpu().numpy()
                                       for c in self.coefficients("cuda"))
            prob = FitProblem(**grid, alpha_E=a_e, beta_E=b_e, alpha_H=np.ones_like(b_h), beta_H=b_h, M_eps=m_e,
                              M_mu=m_h)
        prob.cpml = [CpmlFace(face, b, c, ck) for _, face, b, c, ck in self.cpml]
        for p in range(self.batch):
            mass, flat = self.port_mass(p)
            prob.lumped.append(LumpedPort(np.array([flat]), np.ones(1), np.array([self.dt / mass]), R=R_PORT,
                                          v_src=[self.pulse if q == p else np.zeros(1) for q in range(self.batch)]))
        prob.monitors = [DftMonitor(box, E_COMPONENTS, self.freqs) for box in self.planes]
        prob.e0 = prob.h0 = [None] * self.batch
        return prob


# ---------------------------------------------------------------------------
# The interface
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "modes":
        lap, null, _ = _plane(case, seed)
        return {"kind": kind, "L": lap, "null": null, "n": case["n_modes"]}
    if kind == "serve":
        torch.cuda.init()
        return {"kind": kind, "seed": seed, "case": case}
    if kind == "dispersive":
        prob = dispersive_slab(case["nx"], case["ny"], case["nz"], seed=seed, n_freq=case["n_freq"])
        coef, precision = "native", "single"
    else:
        prob, coef, precision = _Box(case, seed).problem(), case["coef"], case["precision"]
    eng = prob.build_engine(precision)
    if case["stencil"] == "slab":
        eng.configure_stencil("fused", 16)
    if coef != "native":
        eng.set_coefficient_storage(coef)
    eng.reserve_steps(1 << 15)
    return {"kind": kind, "engine": eng, "prob": prob, "steps": case["steps"]}


def _requests(case, seed):
    """Waveguide-section requests as they arrive at the serving loop: sizes
    and inserts from the seed, the channels from the case."""
    rng = np.random.default_rng(seed)
    out = []
    for rid in range(case["requests"]):
        a, b, length = np.array([22.86e-3, 10.16e-3, 40e-3]) * rng.uniform(0.7, 1.3, 3)
        cells = int(np.exp(rng.uniform(np.log(case["cells_lo"]), np.log(case["cells_hi"]))))
        sub, inserts = int(rng.integers(1 << 31)), int(rng.integers(0, 5))

        def build(batch, a=a, b=b, length=length, cells=cells, sub=sub, inserts=inserts):
            return waveguide_section_modal(np.random.default_rng(sub), a=a, b=b, length=length, cells=cells,
                                           n_inserts=inserts, ridged=case["ridged"],
                                           n_modes=(case["modes_in"], case["modes_out"]), n_lumped=case["lumped"],
                                           steps=case["steps"], batch=batch)

        out.append(Request(rid=rid, arrival=0.0, build=build,
                           n_ports=case["modes_in"] + case["modes_out"] + case["lumped"], steps=case["steps"],
                           freqs=np.linspace(7e9, 13e9, case["n_freq"])))
    return out


def run(state):
    kind = state["kind"]
    if kind == "modes":
        lam, vec, _ = sparse_eigs(state["L"], state["n"], state["null"])
        return {"eigenvalues": lam, "modes": vec * np.where(vec[0] < 0.0, -1.0, 1.0)}
    if kind == "serve":
        reqs = _requests(state["case"], state["seed"])
        stats = ServingLoop(records=False).run(reqs)
        # the march is single precision, and so are the scattering parameters kept
        return [r.S.astype(np.complex64) for r in stats.results]
    eng, prob = state["engine"], state["prob"]
    done = eng.steps_done
    end = done + state["steps"]
    res = FitRun(engine=eng, dt=prob.dt, total_time_steps=end, energy_check_interval=100).run(resume_step=done)
    out = {"energy": res.energy_trace["energy"], "fields": [eng.read_fields(b) for b in range(prob.batch)]}
    if kind == "march":
        out["VI"] = [eng.read_vi(b, done, state["steps"]) for b in range(prob.batch)]
        out["dft"] = [eng.read_dft(m, c) for m in range(len(prob.monitors)) for c in E_COMPONENTS]
    else:
        out["energy"] = out["energy"].astype(np.float32)
        out["dft"] = [eng.read_dft(m, "Ex").astype(np.complex64) for m in range(len(prob.monitors))]
    return out


def work(case):
    """Per step: the fields read and written once, the coefficients that are
    not one read once (beta, and alpha of lossy materials).  Absorber states,
    ports and monitors are small beside them and left out."""
    if case["kind"] == "modes":
        n = case["nu"] * case["nv"]
        return {"bytes": 60.0 * n + 8.0 * n * case["n_modes"], "flops": 1000.0 * 10 * n * case["n_modes"]}
    if case["kind"] == "serve":
        updates = case["requests"] * case["steps"] * math.sqrt(case["cells_lo"] * case["cells_hi"])
        sets = case["modes_in"] + case["modes_out"] + case["lumped"]
        return {"bytes": updates * 4.0 * (12 * sets + 6), "flops": updates * sets * 36.0}
    cells = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "dispersive":
        return {"bytes": 4.0 * cells * case["steps"] * (12 + 6 + 3), "flops": 36.0 * cells * case["steps"]}
    word = 8.0 if case["precision"] == "double" else 4.0
    coef = (12 if case["lossy"] else 6) * (2.0 if case["coef"] == "f16" else word)
    return {"bytes": cells * case["steps"] * (12 * word * case["batch"] + coef),
            "flops": 36.0 * cells * case["steps"] * case["batch"]}


def exact(case, seed):
    """The same pass in plain float64 torch (march) or by the separable
    eigenproblem's closed product form (modes)."""
    if case["kind"] == "modes":
        return _plane(case, seed)[2]
    if case["kind"] != "march":
        return None
    return _march64(_Box(case, seed))


# ---------------------------------------------------------------------------
# Port plane: TE Laplacian of a graded rectangle in its symmetric face form
# ---------------------------------------------------------------------------
def _plane(case, seed):
    import scipy.sparse as sp

    rng = np.random.default_rng(seed)
    ones, lows = [], []
    for n, size in ((case["nu"], 22.86e-3), (case["nv"], 10.16e-3)):
        w = rng.uniform(0.8, 1.2, n)
        w *= size / w.sum()
        g = 1.0 / (0.5 * (w[:-1] + w[1:]))
        lap = np.zeros((n, n))
        i = np.arange(n - 1)
        lap[i, i] += g
        lap[i + 1, i + 1] += g
        lap[i, i + 1] -= g
        lap[i + 1, i] -= g
        r = 1.0 / np.sqrt(w)
        ones.append(np.sqrt(w / w.sum()))
        lows.append((lap * r[:, None]) * r[None, :])
    L = sp.kron(sp.csr_matrix(lows[0]), sp.identity(case["nv"])) + sp.kron(sp.identity(case["nu"]),
                                                                           sp.csr_matrix(lows[1]))
    null = np.kron(ones[0], ones[1])[None]
    (lu, vu), (lv, vv) = (np.linalg.eigh(m) for m in lows)
    pairs = sorted((lu[a] + lv[b], a, b) for a in range(5) for b in range(5) if a + b > 0)[:case["n_modes"]]
    vec = np.stack([np.kron(vu[:, a], vv[:, b]) for _, a, b in pairs], axis=1)
    want = {"eigenvalues": np.array([p[0] for p in pairs]), "modes": vec * np.where(vec[0] < 0.0, -1.0, 1.0)}
    return L.tocsr(), null, want


# ---------------------------------------------------------------------------
# Float64 march of a box (the checker's side: plain torch)
# ---------------------------------------------------------------------------
def _back(a, axis):
    """Difference to the previous entry along a spatial axis, with zeros beyond both ends."""
    z = torch.zeros_like(a.narrow(axis + 1, 0, 1))
    return torch.diff(a, dim=axis + 1, prepend=z, append=z)


def _march64(box):
    dev = "cuda"
    B, dt = box.batch, box.dt
    a_e, b_e, m_e, b_h, m_h = box.coefficients(dev)
    lossy = box.sigma is not None or box.pec.size > 0
    zeros = lambda c: torch.zeros((B, *box.shapes[c]), dtype=torch.float64, device=dev)  # noqa: E731
    E, H = [zeros(c) for c in E_COMPONENTS], [zeros(c) for c in ("Hx", "Hy", "Hz")]
    faces = []
    for axis, face, b, c, ck in box.cpml:
        view = [1, 1, 1, 1]
        view[axis + 1] = len(b)
        tab = [torch.as_tensor(np.ascontiguousarray(v), device=dev).view(view) for v in (b, c, ck)]
        faces.append((axis, 0 if face.endswith("min") else box.n[axis] - len(b), len(b), tab))
    psi = {}

    def stretched(key, d, axis):
        for q, (ax, lo, n, (b, c, ck)) in enumerate(faces):
            if ax != axis:
                continue
            s = d.narrow(axis + 1, lo, n)
            p = psi.get((key, q))
            p = c * s if p is None else b * p + c * s
            psi[key, q] = p
            s -= ck * s + p
        return d

    # curl term (component, derivative axis, sign) pairs of each component
    terms = [((2, 1, 1.0), (1, 2, -1.0)), ((0, 2, 1.0), (2, 0, -1.0)), ((1, 0, 1.0), (0, 1, -1.0))]
    ports = [box.port_mass(p) for p in range(B)]
    volt = torch.zeros((box.steps, B, B), dtype=torch.float64, device=dev)
    curr = torch.zeros((box.steps, B, B), dtype=torch.float64, device=dev)
    source = torch.as_tensor(box.pulse, device=dev)
    drive = torch.eye(B, dtype=torch.float64, device=dev)
    widths = [torch.as_tensor(v, device=dev) for v in box.d]
    omega = 2.0 * math.pi * torch.as_tensor(box.freqs, device=dev)
    bins = [torch.zeros((len(box.freqs), *(hi - lo for lo, hi in p)), dtype=torch.complex128, device=dev)
            for p in box.planes for _ in E_COMPONENTS]
    energy = []
    for n in range(box.steps):
        for q in range(3):
            curl = sum(s * stretched(("E", q, c), _back(H[c], ax), ax) for c, ax, s in terms[q])
            if lossy:
                E[q].mul_(a_e[q])
            E[q].add_(curl.mul_(b_e[q]))
        for p in range(B):
            i, j, k = box.port[p]
            mass, _ = ports[p]
            v = E[1][:, i, j, k].clone()
            src = source[n] * drive[p] if n < source.numel() else 0.0 * drive[p]
            cur = (src - v) / (R_PORT + dt / mass)
            E[1][:, i, j, k] += dt / mass * cur
            curr[n, :, p] = cur
        for p in range(B):
            i, j, k = box.port[p]
            volt[n, :, p] = E[1][:, i, j, k]
        for q in range(3):
            curl = sum(s * stretched(("H", q, c), torch.diff(E[c], dim=ax + 1), ax) for c, ax, s in terms[q])
            H[q].sub_(curl.mul_(b_h[q]))
        phase = torch.polar(torch.full_like(omega, dt), omega * (n * dt))[:, None, None, None]
        for m, plane in enumerate(box.planes):
            for q in range(3):
                a = E[q][0]
                for axis in range(3):
                    lo, hi = plane[axis]
                    a = (a.narrow(axis, lo, hi - lo) if axis == q
                         else 0.5 * (a.narrow(axis, lo, hi - lo) + a.narrow(axis, lo + 1, hi - lo)))
                view = [1, 1, 1]
                view[q] = -1
                bins[3 * m + q] += phase * (a / widths[q][plane[q][0]:plane[q][1]].view(view))
        if n % 100 == 0:
            energy.append(float(0.5 * (sum((m * f[0] * f[0]).sum() for m, f in zip(m_e, E))
                                       + sum((m * f[0] * f[0]).sum() for m, f in zip(m_h, H)))))
    V, I = volt.permute(1, 0, 2).cpu().numpy(), curr.permute(1, 0, 2).cpu().numpy()
    flat = lambda F, b: torch.cat([f[b].reshape(-1) for f in F])  # noqa: E731
    return {"energy": np.array(energy), "fields": [(flat(E, b), flat(H, b)) for b in range(B)],
            "VI": [(V[b], I[b]) for b in range(B)], "dft": bins}
