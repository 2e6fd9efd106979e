"""Measured cases: the calls a user of this framework makes, over the sizes they are made at.

A case names a family and its sizes; its inputs are made from a seed alone.

residual    one SCF residual evaluation x -> f on device vectors (System.residual_device): the inner call of
            every iteration a program keeps for itself
gradient    J^T w at x, from device vectors (sfgpu_vjp) or from host arrays (System.vjp): the gradient of a
            loss on the residual, L-BFGS, chi sensitivities
tangent     J v at x on device vectors (sfgpu_jvp): Newton-Krylov and GMRES
solve       one system iterated by Pure_DIIS to convergence (System.solve) from host guesses
batch       a parameter sweep, many systems in one launch (BatchSolver.solve) from host guesses

Systems: "flat1d" (homopolymer at an adsorbing wall, Lat1DFlat1stO), "cyl2d" (diblock around a particle on the
axis of a cylinder, Lat2DCyl1stO), "flat2d_semi" (semiflexible chains, Lat2D2ndO), "melt3d" (periodic diblock
melt, Lat3D1stO) and "brush3d" (semiflexible grafted brush, Lat3D2ndO).
"""
import math

import numpy as np
import torch

from field_b200 import configs
from field_b200.batch import BatchSolver
from field_b200.desc import (BOUND_MIRROR1, BOUND_PERIODIC, GEOM_CYLINDRICAL, GEOM_FLAT, Lattice, Molecule, MOL_FREE,
                             MOL_SOLVENT, Segment, SEG_FROZEN, SystemSpec)
from field_b200.system import System

TOL = 1e-11          # solves: tight, so that the converged x is the system's and not the iteration's
MAXIT = 3000


def listed():
    return [
        # the 1D adsorption system every introduction starts with: the smallest call, latency and launches
        {"name": "residual_flat1d", "family": "residual", "system": "flat1d", "n": 100, "N": 100},
        # the cylindrical micelle / colloid lattice of the benchmark, one evaluation of a diblock
        {"name": "residual_cyl2d", "family": "residual", "system": "cyl2d", "nx": 128, "ny": 128, "N": 40},
        # semiflexible chains on a 2D lattice (the Markov option), an uneven box
        {"name": "residual_flat2d_semi", "family": "residual", "system": "flat2d_semi", "nx": 61, "ny": 77, "N": 100},
        # the block copolymer melt in a 3D box at full size: bandwidth
        {"name": "residual_melt3d", "family": "residual", "system": "melt3d", "nx": 128, "ny": 128, "nz": 128,
         "N": 100},
        # a grafted semiflexible brush in a 3D box at full size: six direction components, 9 GB of chain storage
        {"name": "residual_brush3d", "family": "residual", "system": "brush3d", "n": 96, "nz": 96, "N": 200},
        # gradient through the cylinder system from host arrays: one step of a host-side optimiser
        {"name": "gradient_cyl2d_host", "family": "gradient", "system": "cyl2d", "nx": 128, "ny": 128, "N": 40,
         "host": True},
        # gradient through the full-size melt on device vectors
        {"name": "gradient_melt3d", "family": "gradient", "system": "melt3d", "nx": 128, "ny": 128, "nz": 128,
         "N": 100, "host": False},
        # Jacobian product of a melt in an uneven box with odd sides
        {"name": "tangent_melt3d", "family": "tangent", "system": "melt3d", "nx": 90, "ny": 75, "nz": 61, "N": 64},
        # one 1D calculation from scratch: an input file's worth of work
        {"name": "solve_flat1d", "family": "solve", "system": "flat1d", "n": 200, "N": 200, "m": 5},
        # one 2D calculation from scratch
        {"name": "solve_cyl2d", "family": "solve", "system": "cyl2d", "nx": 128, "ny": 128, "N": 40, "m": 10},
        # a sweep of uneven 1D calculations (layers 50..400, N 20..1000)
        {"name": "batch_flat1d", "family": "batch", "system": "flat1d", "count": 256, "n": 400, "N": 1000, "m": 5},
        # a sweep on the benchmark's 2D lattice, two instances per SM
        {"name": "batch_cyl2d", "family": "batch", "system": "cyl2d", "count": 296, "nx": 128, "ny": 128, "N": 40,
         "m": 10},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.randrange(10)
    if kind == 0:
        return {"family": "residual", "system": "flat1d", "n": _log(rng, 40, 500), "N": _log(rng, 20, 1000)}
    if kind == 1:
        return {"family": "residual", "system": "cyl2d", "nx": _log(rng, 24, 200), "ny": _log(rng, 24, 200),
                "N": _log(rng, 10, 200)}
    if kind == 2:
        return {"family": "residual", "system": "flat2d_semi", "nx": _log(rng, 20, 160), "ny": _log(rng, 20, 160),
                "N": _log(rng, 10, 200)}
    if kind == 3:
        return {"family": "residual", "system": "melt3d", "nx": _log(rng, 16, 128), "ny": _log(rng, 16, 128),
                "nz": _log(rng, 16, 128), "N": _log(rng, 10, 100)}
    if kind == 4:
        return {"family": "residual", "system": "brush3d", "n": _log(rng, 16, 96), "nz": _log(rng, 16, 96),
                "N": _log(rng, 10, 200)}
    if kind == 5:
        return {"family": "gradient", "system": "cyl2d", "nx": _log(rng, 24, 200), "ny": _log(rng, 24, 200),
                "N": _log(rng, 10, 100), "host": rng.random() < 0.5}
    if kind == 6:
        return {"family": rng.choice(["gradient", "tangent"]), "system": "melt3d", "nx": _log(rng, 16, 128),
                "ny": _log(rng, 16, 128), "nz": _log(rng, 16, 128), "N": _log(rng, 10, 100), "host": False}
    if kind == 7:
        return {"family": "solve", "system": "flat1d", "n": _log(rng, 50, 400), "N": _log(rng, 20, 1000), "m": 5}
    if kind == 8:
        return {"family": "solve", "system": "cyl2d", "nx": _log(rng, 32, 128), "ny": _log(rng, 32, 128),
                "N": _log(rng, 10, 60), "m": 10}
    if rng.random() < 0.5:
        return {"family": "batch", "system": "flat1d", "count": _log(rng, 16, 256), "n": _log(rng, 80, 400),
                "N": _log(rng, 50, 1000), "m": 5}
    return {"family": "batch", "system": "cyl2d", "count": _log(rng, 8, 296), "nx": _log(rng, 32, 128),
            "ny": _log(rng, 32, 128), "N": _log(rng, 10, 40), "m": 10}


# ---------------------------------------------------------------------------
# systems: parameters of the instances, their specs and their inputs
def _params(case, seed):
    """Sizes (the case's alone) and interaction parameters (the seed's) of every instance of a case."""
    rng = np.random.default_rng(seed)
    sizes = np.random.default_rng(case["N"] + 7919 * case.get("count", 1))
    count = case.get("count", 1)
    out = []
    for _ in range(count):
        p = dict(case)
        if case["system"] == "flat1d":
            if case["family"] == "batch":      # uneven instances up to the case's sizes
                p["n"] = int(sizes.integers(max(20, case["n"] // 8), case["n"] + 1))
                p["N"] = int(round(math.exp(sizes.uniform(math.log(max(10, case["N"] // 50)), math.log(case["N"])))))
            p["phib"] = float(math.exp(rng.uniform(math.log(1e-4), math.log(5e-2))))
            p["chi_aw"] = float(rng.uniform(0.0, 0.45))
            p["chi_as"] = float(rng.uniform(-1.5, -0.5))
        elif case["system"] == "cyl2d":
            p["phib"] = float(math.exp(rng.uniform(math.log(1e-3), math.log(1e-2))))
            p["chi_aw"] = float(rng.uniform(0.2, 0.5))
            p["chi_as"] = float(rng.uniform(-1.5, -0.8))
            p["R"] = 6.0
        elif case["system"] == "flat2d_semi":
            p["phib"] = float(rng.uniform(0.005, 0.02))
            p["chi_aw"], p["chi_as"], p["S"] = 0.4, -1.0, 0.5
        elif case["system"] == "melt3d":
            p["chi_ab"] = 20.0 / case["N"]
        else:
            p["chi_aw"], p["S"], p["sigma"] = 0.3, 0.2, 0.05
        out.append(p)
    return out


def _split(N):
    return N // 2, N - N // 2


def _wall_chi(p):
    """Segments S, A, B, W: A adsorbs on S, A and W repel."""
    chi = np.zeros((4, 4))
    chi[0, 1] = chi[1, 0] = p["chi_as"]
    chi[1, 3] = chi[3, 1] = p["chi_aw"]
    return chi


def _particle(nx, ny, R):
    x, y = np.meshgrid(np.arange(nx + 2) - 0.5, np.arange(ny + 2) - (ny + 1) / 2.0, indexing="ij")
    return (x * x + y * y < R * R).astype(float)


def _spec(p, seed):
    s = p["system"]
    if s == "flat1d":
        return configs.flat_adsorption(p["n"], p["N"], p["phib"], p["chi_aw"], p["chi_as"])[0]
    if s in ("cyl2d", "flat2d_semi"):
        cyl = s == "cyl2d"
        lat = Lattice(2, [p["nx"], p["ny"], 0], [BOUND_MIRROR1] * 2 + [0], [BOUND_MIRROR1] * 2 + [0],
                      geometry=GEOM_CYLINDRICAL if cyl else GEOM_FLAT, order=1 if cyl else 2, lam=1.0 / 6.0)
        segs = [Segment("S", SEG_FROZEN, _particle(p["nx"], p["ny"], p.get("R", 5.0)).reshape(-1)), Segment("A"),
                Segment("B"), Segment("W")]
        nA, nB = _split(p["N"])
        mols = [Molecule("AB", [(1, nA), (2, nB)], MOL_FREE, phibulk=p["phib"]), Molecule("W", [(3, 1)], MOL_SOLVENT)]
        return SystemSpec(lat, segs, _wall_chi(p), mols, pf=None if cyl else np.full((4, 4), p["S"]))
    if s == "melt3d":
        lat = Lattice(3, [p["nx"], p["ny"], p["nz"]], [BOUND_PERIODIC] * 3, [BOUND_PERIODIC] * 3)
        nA, nB = _split(p["N"])
        return SystemSpec(lat, [Segment("A"), Segment("B")], np.array([[0.0, p["chi_ab"]], [p["chi_ab"], 0.0]]),
                          [Molecule("AB", [(0, nA), (1, nB)], MOL_SOLVENT)])
    return configs.brush3d(n=p["n"], N=p["N"], sigma=p["sigma"], chi=p["chi_aw"], S=p["S"], seed=seed, nz=p["nz"])[0]


def _shape(p):
    s = p["system"]
    if s == "flat1d":
        return (p["n"],)
    if s in ("cyl2d", "flat2d_semi"):
        return (p["nx"], p["ny"])
    return (p["nx"], p["ny"], p["nz"]) if s == "melt3d" else (p["n"], p["n"], p["nz"])


def _field(nvar, seed, amp=0.1):
    """Potentials as an iteration meets them: a long wave along the sites and noise on every value."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    x = torch.randn(nvar, generator=g, device="cuda", dtype=torch.float64) * amp
    k = torch.rand(1, generator=g, device="cuda", dtype=torch.float64) * 6 + 2
    return x + 0.3 * torch.cos(torch.arange(nvar, device="cuda", dtype=torch.float64) * (k * math.pi / nvar))


def _weights(nvar, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 77777)
    return torch.randn(nvar, generator=g, device="cuda", dtype=torch.float64)


def prepare(case, seed):
    ps = _params(case, seed)
    st = {"case": case}
    if case["family"] == "batch":
        st["solver"] = BatchSolver([_spec(p, seed) for p in ps], m=case["m"], eta=0.1)
        st["x0"] = np.zeros(st["solver"].total)
        return st
    s = System(_spec(ps[0], seed))
    s.use_stream(torch.cuda.current_stream().cuda_stream)
    st["system"] = s
    if case["family"] == "solve":
        st["x0"] = np.zeros(s.nvar)
        return st
    st["x"] = _field(s.nvar, seed)
    if case["family"] in ("gradient", "tangent"):
        st["v"] = _weights(s.nvar, seed)
    if case.get("host"):
        st["x"], st["v"] = st["x"].cpu().numpy(), st["v"].cpu().numpy()
    else:
        st["f"], st["out"] = torch.empty_like(st["x"]), torch.empty_like(st["x"])
    return st


def run(state):
    case, fam = state["case"], state["case"]["family"]
    if fam == "batch":
        r = state["solver"].solve(state["x0"], tol=TOL, maxit=MAXIT)
        return {"x": r.x, "status": r.status}
    s = state["system"]
    if fam == "solve":
        r = s.solve(state["x0"], tol=TOL, maxit=MAXIT, m=case["m"], eta=0.1)
        return {"x": r.x, "status": r.status}
    if case.get("host"):
        f, g = s.vjp(state["x"], state["v"])
        return {"f": f, "g": g}
    x, f = state["x"], state["f"]
    if fam == "residual":
        s.residual_device(x.data_ptr(), f.data_ptr())
        return {"f": f}
    call = s.lib.sfgpu_vjp if fam == "gradient" else s.lib.sfgpu_jvp
    rc = call(s.h, x.data_ptr(), state["v"].data_ptr(), f.data_ptr(), state["out"].data_ptr())
    if rc:
        raise RuntimeError(f"status {rc}")
    return {"f": f, "g": state["out"]}


# iterations that Pure_DIIS takes on these systems from x = 0 at the tolerance above, about
ITERATIONS = 70


def work(case):
    """Bytes: inputs and outputs once; on the 3D lattices, whose chains exceed every on-chip memory, the chain's
    slices written once by one sweep and read once by the other (twice for a gradient or a Jacobian product).
    Flops: the two propagator sweeps and the composition, per site, component and segment."""
    tot_b = tot_f = 0.0
    for p in _params(case, 1):
        M = float(np.prod(_shape(p)))
        K = {"flat2d_semi": 5, "brush3d": 6}.get(p["system"], 1)
        nclass = {"flat1d": 2, "cyl2d": 3, "flat2d_semi": 3, "melt3d": 2, "brush3d": 3}[p["system"]]
        per = {"flat1d": 8, "cyl2d": 14, "flat2d_semi": 10, "melt3d": 9, "brush3d": 12}[p["system"]]
        sweeps = 2 if case["family"] in ("gradient", "tangent") else 1
        nvar = M * nclass
        fl = sweeps * 2.0 * p["N"] * M * K * per + 40 * nvar
        by = 8 * 2 * nvar * sweeps
        if len(_shape(p)) == 3:
            by += sweeps * 16 * p["N"] * K * M
        if case["family"] in ("solve", "batch"):
            fl = ITERATIONS * (fl + 6 * (case["m"] + 2) * nvar)
        tot_b += by
        tot_f += fl
    return {"bytes": tot_b, "flops": tot_f}


# ---------------------------------------------------------------------------
# the same quantities in plain torch, 64 bits: fields are (instance, interior sites)
def _shift(a, dim, step, periodic, lo=None):
    """Values one site away (step -1: the lower neighbour); lo: the value below the first site (None: the first
    site's own, mirror1); above the last one mirror1."""
    if periodic:
        return torch.roll(a, -step, dim)
    n = a.shape[dim]
    if step > 0:
        return torch.cat([a.narrow(dim, 1, n - 1), a.narrow(dim, n - 1, 1)], dim)
    edge = a.narrow(dim, 0, 1)
    edge = edge if lo is None else torch.full_like(edge, lo)
    return torch.cat([edge, a.narrow(dim, 0, n - 1)], dim)


class _Exact:
    def __init__(self, case, ps, seed):
        p = ps[0]
        self.p, self.sys, self.shape, self.N = p, p["system"], _shape(p), p["N"]
        dev = dict(device="cuda", dtype=torch.float64)
        self.per = self.sys == "melt3d"
        self.wall = self.sys == "flat1d"
        B, one = len(ps), (1,) * len(self.shape)
        col = lambda k: torch.tensor([q[k] for q in ps], **dev).reshape((B,) + one)  # noqa: E731
        nA, nB = _split(self.N)
        self.chi, self.frozen = {}, None
        if self.sys == "flat1d":
            self.names, self.chain = ["A", "W"], ["A"] * self.N
        elif self.sys in ("cyl2d", "flat2d_semi"):
            self.names, self.chain = ["A", "B", "W"], ["A"] * nA + ["B"] * nB
            m = _particle(p["nx"], p["ny"], p.get("R", 5.0))[1:-1, 1:-1]
            self.frozen = torch.tensor(m, **dev)[None]
        elif self.sys == "melt3d":
            self.names, self.chain = ["A", "B"], ["A"] * nA + ["B"] * nB
        else:
            self.names, self.chain = ["X", "A", "W"], ["X"] + ["A"] * (self.N - 1)
            n = p["n"]
            ng = int(round(p["sigma"] * n * n))
            at = np.random.default_rng(seed).choice(n * n, size=ng, replace=False)
            m = np.zeros(self.shape)
            m[at // n, at % n, 0] = 1.0
            self.pinned, self.theta = torch.tensor(m, **dev)[None], float(ng * self.N)
        for a, b, k in (("A", "W", "chi_aw"), ("A", "S", "chi_as"), ("A", "B", "chi_ab")):
            if k in p:
                self.chi[a, b] = self.chi[b, a] = col(k)
        self.phib = col("phib") if "phib" in p else None
        if self.sys == "cyl2d":
            # a ring of layers x-1 .. x: pi (2x - 1) sites, 2 pi x / 6 bonds outwards
            x = torch.arange(1, self.shape[0] + 1, **dev)
            self.lp = (2 * x / 6 / (2 * x - 1)).reshape(1, -1, 1)
            self.lm = (2 * (x - 1) / 6 / (2 * x - 1)).reshape(1, -1, 1)
        self.free = None if self.frozen is None else (self.frozen == 0)[0]

    def nb(self, a, axis, step, lo=0.0):
        return _shift(a, axis + 1, step, self.per, lo if self.wall else None)

    def mean(self, a, lo=0.0):
        """Contact average; the first-order step is G times it."""
        if len(self.shape) == 1:
            return a + (self.nb(a, 0, -1, lo) - 2 * a + self.nb(a, 0, 1)) / 6
        if self.sys == "cyl2d":
            return (a + self.lm * (self.nb(a, 0, -1) - a) + self.lp * (self.nb(a, 0, 1) - a)
                    + (self.nb(a, 1, -1) + self.nb(a, 1, 1) - 2 * a) / 6)
        tot = sum(self.nb(a, d, s) for d in range(len(self.shape)) for s in (-1, 1))
        return tot / 6 + (a / 3 if len(self.shape) == 2 else 0)

    # second order: a propagator is a dict of bond directions (axis, sign); a homogeneous axis is one lumped entry
    def dirs(self):
        d = [(a, s) for a in range(len(self.shape)) for s in (1, -1)]
        return d + ([("z", 1)] if len(self.shape) == 2 else [])

    def mult(self, k):
        return 2.0 if k[0] == "z" else 1.0

    def weight(self, k, kp):
        S = self.p["S"]
        if k == kp:
            return S                      # the lumped z group: straight on S, back 0
        if k[0] == kp[0]:
            return 0.0
        return self.mult(kp) * (1 - S) / 4

    def take(self, gs, kp, axis, step):
        """Component kp one site away; across a mirror the axis' directions change places."""
        a = gs[kp]
        got = self.nb(a, axis, step)
        if kp[0] != axis:
            return got
        n = a.shape[axis + 1]
        other = gs[(axis, -kp[1])].narrow(axis + 1, n - 1 if step > 0 else 0, 1)
        if step > 0:
            return torch.cat([got.narrow(axis + 1, 0, n - 1), other], axis + 1)
        return torch.cat([other, got.narrow(axis + 1, 1, n - 1)], axis + 1)

    def step(self, g, gs, back):
        if not isinstance(gs, dict):
            return g * self.mean(gs)
        out = {}
        if not back:
            for k in gs:
                src = {kp: (gs[kp] if k[0] == "z" else self.take(gs, kp, k[0], -k[1])) for kp in gs
                       if self.weight(k, kp)}
                out[k] = g * sum(self.weight(k, kp) * v for kp, v in src.items())
            return out
        v = {kp: (gs[kp] if kp[0] == "z" else self.take(gs, kp, kp[0], kp[1])) for kp in gs}
        for k in gs:
            out[k] = g * sum(self.weight(k, kp) * v[kp] for kp in gs if self.weight(k, kp))
        return out

    def dot(self, a, b):
        return sum(self.mult(k) * a[k] * b[k] for k in a) if isinstance(a, dict) else a * b

    def residual(self, x):
        """x: (instance, values) in the iteration's packing (site-major, one value per segment type)."""
        B, nc = x.shape[0], len(self.names)
        u = x.reshape(B, -1, nc)
        if self.free is not None:
            full = torch.zeros(B, int(np.prod(self.shape)), nc, device=x.device, dtype=x.dtype)
            at = torch.nonzero(self.free.reshape(-1))[:, 0]
            u = full.index_copy(1, at, u)
        u = u.reshape((B,) + self.shape + (nc,))
        G = {n: torch.exp(-u[..., i]) for i, n in enumerate(self.names)}
        Gs = dict(G)
        if self.frozen is not None:
            Gs = {n: torch.where(self.free[None], g, torch.zeros_like(g)) for n, g in G.items()}
        if "X" in Gs:
            Gs["X"] = G["X"] * self.pinned
        second = self.sys in ("brush3d", "flat2d_semi")
        rep = (lambda g: {k: g for k in self.dirs()}) if second else (lambda g: g)
        fw = [rep(Gs[self.chain[0]])]
        for s in self.chain[1:]:
            fw.append(self.step(Gs[s], fw[-1], False))
        back = rep(Gs[self.chain[-1]])
        raw = {self.chain[-1]: self.dot(back, fw[-1])}
        for t in range(self.N - 2, -1, -1):
            s = self.chain[t]
            back = self.step(Gs[s], back, True)
            c = self.dot(back, fw[t])
            raw[s] = raw[s] + c if s in raw else c
        N = float(self.N)
        if self.sys == "brush3d":
            norm = self.theta / N / sum(b.sum() for b in back.values())
            bulk = {"X": 0.0, "A": 0.0, "W": 1.0}
        elif self.sys == "melt3d":
            norm = 1.0 / N
            bulk = {n: self.chain.count(n) / N for n in self.names}
        else:
            norm = self.phib / N / (6 if second else 1)
            bulk = {n: self.phib * (self.chain.count(n) / N) for n in set(self.chain)}
            bulk["W"] = 1 - self.phib
        phi = {n: norm * torch.where(Gs[n] > 0, r / torch.where(Gs[n] > 0, Gs[n], torch.ones_like(r)),
                                     torch.zeros_like(r)) for n, r in raw.items()}
        if "W" in self.names:
            phi["W"] = Gs["W"] * bulk["W"]
        tot = sum(phi.values())
        rho = {n: self.mean(q) for n, q in phi.items()}
        if self.frozen is not None:
            tot = tot + self.frozen
            rho["S"] = self.mean(self.frozen)
        if self.wall:
            rho["S"] = self.mean(torch.zeros_like(tot), 1.0)
        up = []
        for i, n in enumerate(self.names):
            c = sum((self.chi[n, o] * rho[o] for o in rho if (n, o) in self.chi), torch.zeros_like(tot))
            b = sum((self.chi[n, o] * bulk[o] for o in bulk if (n, o) in self.chi), torch.zeros_like(tot))
            up.append(u[..., i] - c / tot + b)
        up = torch.stack(up, -1)
        f = -1 + 1 / tot[..., None] + up - up.mean(-1, keepdim=True)
        f = f.reshape(B, -1, nc)
        return (f if self.free is None else f[:, at]).reshape(B, -1)

    def solve(self, nvar, B):
        """Anderson mixing to a residual well below the cases' tolerance."""
        x = torch.zeros(B, nvar, device="cuda", dtype=torch.float64)
        X, F = [], []
        for _ in range(500):
            f = self.residual(x)
            if float(f.norm(dim=1).max()) < 1e-12:
                break
            X.append(x)
            F.append(f)
            X, F = X[-11:], F[-11:]
            x = x - 0.1 * f
            if len(F) > 1:
                dF = torch.stack([F[i + 1] - F[i] for i in range(len(F) - 1)], -1)
                dX = torch.stack([X[i + 1] - X[i] for i in range(len(X) - 1)], -1)
                A = dF.transpose(1, 2) @ dF
                sc = A.diagonal(dim1=1, dim2=2).sqrt().clamp_min(1e-300)
                A = A / sc[:, :, None] / sc[:, None, :]
                b = (dF.transpose(1, 2) @ f[:, :, None])[..., 0] / sc
                g = (torch.linalg.pinv(A, rtol=1e-14, hermitian=True) @ b[:, :, None])[..., 0] / sc
                x = x - ((dX - 0.1 * dF) @ g[:, :, None])[..., 0]
        return x


def exact(case, seed):
    ps = _params(case, seed)
    if case["family"] == "batch" and case["system"] == "flat1d":
        return None                      # uneven chains one after another: minutes
    e = _Exact(case, ps, seed)
    nsites = int(np.prod(e.shape)) if e.free is None else int(e.free.sum())
    nvar = nsites * len(e.names)
    if case["family"] in ("solve", "batch"):
        with torch.no_grad():
            x = torch.cat([_Exact(case, ps[i:i + 64], seed).solve(nvar, len(ps[i:i + 64]))
                           for i in range(0, len(ps), 64)])
        return {"x": x.reshape(-1).cpu().numpy(), "status": None}
    x = _field(nvar, seed)[None]
    if case["family"] == "residual":
        with torch.no_grad():
            return {"f": e.residual(x)[0]}
    v = _weights(nvar, seed)[None]
    if case["family"] == "tangent":
        f, g = torch.func.jvp(e.residual, (x,), (v,))
        return {"f": f[0], "g": g[0]}
    x.requires_grad_(True)
    f = e.residual(x)
    (g,) = torch.autograd.grad(f, x, v)
    f, g = f[0].detach(), g[0]
    return {"f": f.cpu().numpy(), "g": g.cpu().numpy()} if case.get("host") else {"f": f, "g": g}
