"""Performance cases of the solid hot path: what a user's program asks of
libfastgpu through fast_b200.gpu.GpuSystem, from one small linear-static step
to the 1.6-million-equation box, with the inputs, one pass and a 64-bit value
of its results (plain torch, no library code) for each.

Families
  static    new moduli -> assemble K -> solve K u = f    (linear-static controller)
  tied      the same on a multi-block model with tied interfaces and B-splines
  assemble  new coordinates and moduli -> K and M, one product with each
  tangent   a displacement state -> TL tangent, internal force, one product
  newton    load-control Newton on a total-Lagrangian plate
  newmark   linear transient response under a step load
  ensemble  many independent cantilevers: assemble and solve in one batch

Meshes are boxes of hex8 or hex20 elements whose nodes are moved by a few
percent of their spacing (no two elements alike), with a lognormal Young's
modulus per element; load vectors are made here, per equation.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from fast_b200 import decks, gpu

PREC = {"fp64": gpu.PREC_FP64, "mixed": gpu.PREC_MIXED}


# -------------------------------------------------------------------- cases

def _static(name, kind, n, L, clamp, precision, assembly, tol):
    return {"name": name, "family": "static", "kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "lx": L[0],
            "ly": L[1], "lz": L[2], "clamp": clamp, "precision": precision, "assembly": assembly, "tol": tol}


def _cubes(n, h=1.0 / 16):
    return tuple(k * h for k in n)


def listed():
    return [
        # the plain linear-static cantilever: the smallest call, launches and host waits count
        _static("static hex8 20x4x4", "hex8", (20, 4, 4), (10.0, 1.0, 1.0), 0, "fp64", "fp64", 1e-12),
        # a small ragged quadratic model in plain FP64 (the reference's algorithm)
        _static("static hex20 13x9x7", "hex20", (13, 9, 7), _cubes((13, 9, 7)), 2, "fp64", "fp64", 1e-10),
        # quadratic model of ordinary size assembled on the tensor cores, mixed-precision solve
        _static("static hex20 26x25x14 tf32", "hex20", (26, 25, 14), _cubes((26, 25, 14)), 2, "mixed", "tf32", 1e-10),
        # linear elements, ordinary size, mixed precision
        _static("static hex8 61x47x33", "hex8", (61, 47, 33), _cubes((61, 47, 33)), 2, "mixed", "fp64", 1e-10),
        # quadratic elements, larger, plain FP64
        _static("static hex20 40x33x21", "hex20", (40, 33, 21), _cubes((40, 33, 21)), 2, "fp64", "fp64", 1e-10),
        # the headline workload's size: 131,072 hex20 elements, mixed precision
        _static("static hex20 64x64x32", "hex20", (64, 64, 32), _cubes((64, 64, 32)), 2, "mixed", "fp64", 1e-10),
        # hex8 + hex20 + B-spline p=2 and p=3 blocks joined by tied interfaces
        {"name": "tied column", "family": "tied", "h8": 20, "h20": 12, "p2": 16, "p3": 12, "precision": "mixed",
         "tol": 1e-10},
        # re-assembly alone, as a controller does when geometry and material change
        {"name": "assemble hex20 40x39x21", "family": "assemble", "kind": "hex20", "nx": 40, "ny": 39, "nz": 21},
        # one evaluation of a Newton iteration: tangent, internal force, product
        {"name": "tangent hex8 81x79x6", "family": "tangent", "kind": "hex8", "nx": 81, "ny": 79, "nz": 6},
        # Newton on the TL plate, mixed-precision inner solves, secant starts
        {"name": "newton hex8 40x40x4", "family": "newton", "nx": 40, "ny": 40, "nz": 4, "steps": 6,
         "precision": "mixed", "predictor": 1},
        # transient response: mass and stiffness, warm-started solves
        {"name": "newmark hex20 24x23x12", "family": "newmark", "kind": "hex20", "nx": 24, "ny": 23, "nz": 12,
         "steps": 12, "precision": "mixed"},
        # independent uneven problems in one launch
        {"name": "ensemble 256", "family": "ensemble", "count": 256, "nmin": 6, "nmax": 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    """Box dimensions of about lo..hi elements, each direction ragged."""
    m = _log(rng, lo, hi) ** (1.0 / 3)
    return tuple(max(2, int(round(m * rng.uniform(0.7, 1.35)))) for _ in range(3))


def draw(rng):
    fam = rng.choice(["static"] * 6 + ["tied", "assemble", "tangent", "newton", "newmark", "ensemble"])
    if fam == "static":
        kind = rng.choice(["hex8", "hex20"])
        n = _box(rng, 200, 250_000 if kind == "hex8" else 45_000)
        precision = rng.choice(["fp64", "mixed"])
        assembly = "tf32" if precision == "mixed" and rng.random() < 0.3 else "fp64"
        c = _static("", kind, n, _cubes(n), rng.choice([0, 2]), precision, assembly, 1e-10)
        del c["name"]
        return c
    if fam == "tied":
        s = rng.uniform(0.45, 1.4)
        k = lambda v: max(4, int(round(v * s * rng.uniform(0.85, 1.15))))  # noqa: E731
        return {"family": fam, "h8": k(20), "h20": k(12), "p2": k(16), "p3": k(12),
                "precision": rng.choice(["fp64", "mixed"]), "tol": 1e-10}
    if fam in ("assemble", "tangent"):
        kind = rng.choice(["hex8", "hex20"])
        n = _box(rng, 300, 120_000 if kind == "hex8" else 40_000)
        return {"family": fam, "kind": kind, "nx": n[0], "ny": n[1], "nz": n[2]}
    if fam == "newton":
        return {"family": fam, "nx": _log(rng, 9, 44), "ny": _log(rng, 9, 44), "nz": rng.randint(2, 5),
                "steps": rng.randint(2, 6), "precision": rng.choice(["fp64", "mixed"]),
                "predictor": rng.choice([0, 1])}
    if fam == "newmark":
        kind = rng.choice(["hex8", "hex20"])
        n = _box(rng, 300, 40_000 if kind == "hex8" else 9_000)
        return {"family": fam, "kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "steps": rng.randint(4, 14),
                "precision": rng.choice(["fp64", "mixed"])}
    lo = rng.randint(3, 9)
    return {"family": fam, "count": _log(rng, 8, 256), "nmin": lo, "nmax": lo + rng.randint(3, 11)}


# ------------------------------------------------------------------- inputs

@functools.lru_cache(maxsize=6)
def _mesh(kind, n, L):
    return decks.box_mesh(kind, n, L)


@functools.lru_cache(maxsize=2)
def _column(h8, h20, p2, p3):
    half = lambda v: max(2, v // 2)  # noqa: E731
    return decks.tied_column((h8, h8, half(h8)), (h20, h20, half(h20)), (p2, p2, max(2, p2 // 4)),
                             (p3, p3, max(2, p3 // 4)))


def _box_deck(kind, n, L, rng, clamp=2, sides=False, jitter=0.05, sigma=0.5, rho=None, tl=False):
    """A box with moved nodes and lognormal moduli; the low face of axis
    `clamp` (or, with sides, the four side faces) fixed."""
    X, conn, _ = _mesh(kind, n, L)
    h = np.asarray(L) / np.asarray(n) / (2 if kind == "hex20" else 1)
    Y = X + rng.uniform(-jitter, jitter, X.shape) * h
    fixed = np.zeros(X.shape, bool)
    at = lambda d, v: np.abs(X[:, d] - v) < 1e-9  # noqa: E731
    fixed[at(0, 0) | at(0, L[0]) | at(1, 0) | at(1, L[1]) if sides else at(clamp, 0)] = True
    ne = len(conn)
    loaded = at(2, L[2]) if sides else at(clamp, L[clamp])
    E = 1000.0 * np.exp(sigma * rng.standard_normal(ne))
    g = 2 if kind == "hex8" else 3
    d = decks.Deck(kind, Y, conn, E, np.full(ne, 0.3), (g, g, g), fixed, matrix_type="sparse",
                   rho=None if rho is None else np.full(ne, rho), total_lagrangian=tl)
    return d, loaded


def _face_load(deck, loaded, rng, total):
    """Nodal forces on the loaded face, uneven from node to node."""
    eq = deck.node_eq()
    f = np.zeros(int(eq.max()))
    for k in range(3):
        q = eq[loaded, k]
        q = q[q > 0] - 1
        f[q] = total[k] * (1.0 + 0.3 * rng.standard_normal(len(q))) / max(1, int(loaded.sum()))
    return f


def _inputs(c, seed):
    """(deck, dict of the pass's host arrays) from the seed alone."""
    rng = np.random.default_rng([seed, 7])
    fam = c["family"]
    if fam == "tied":
        d = _column(c["h8"], c["h20"], c["p2"], c["p3"])
        E = [1000.0 * np.exp(0.3 * rng.standard_normal(b.num_elems)) for b in d.buckets()]
        f = decks.nodal_load_vector(d)
        return d, {"E": E, "f": f * (1.0 + 0.3 * rng.standard_normal(f.shape))}
    if fam == "ensemble":
        ns = np.random.default_rng(c["count"]).integers(c["nmin"], c["nmax"] + 1, size=c["count"])
        members, f = [], []
        for n in ns:
            n = int(n)
            m, loaded = _box_deck("hex8", (2 * n, n, n), (2.0, 1.0, 1.0), rng, clamp=0)
            members.append(m)
            f.append(_face_load(m, loaded, rng, rng.standard_normal(3)))
        d, noff, _ = decks.concat_decks(members)
        return d, {"E": d.E.copy(), "f": np.concatenate(f), "noff": noff}
    n = (c["nx"], c["ny"], c["nz"])
    if fam == "static":
        d, loaded = _box_deck(c["kind"], n, (c["lx"], c["ly"], c["lz"]), rng, clamp=c["clamp"])
        return d, {"E": d.E.copy(), "f": _face_load(d, loaded, rng, (0.3, -0.2, -1.0))}
    if fam == "assemble":
        d, _ = _box_deck(c["kind"], n, _cubes(n), rng, rho=1e-3)
        return d, {"X": d.coords.copy(), "E": d.E.copy(), "x": rng.standard_normal(d.num_eq())}
    if fam == "tangent":
        d, _ = _box_deck(c["kind"], n, _cubes(n), rng, sides=True, sigma=0.1, tl=True)
        u = 0.01 / 16 * rng.standard_normal(d.num_eq())
        return d, {"u": u, "x": rng.standard_normal(d.num_eq())}
    if fam == "newton":
        L = (n[0] / 4, n[1] / 4, n[2] / 4)
        d, loaded = _box_deck("hex8", n, L, rng, sides=True, jitter=0.02, sigma=0.1, tl=True)
        return d, {"q": _face_load(d, loaded, rng, (0.0, 0.0, -0.35 * c["steps"] * L[0] * L[1]))}
    d, loaded = _box_deck(c["kind"], n, _cubes(n), rng, rho=1e-3)
    return d, {"f": _face_load(d, loaded, rng, (0.0, 0.0, -1.0))}


def prepare(case, seed):
    d, a = _inputs(case, seed)
    S = gpu.GpuSystem(0)
    S.upload(d)
    if case["family"] == "ensemble":
        S.set_problems(a["noff"])
    return {"case": case, "S": S, **a}


# ----------------------------------------------------------------- one pass

_NEWMARK_DT = 2e-3


def run(s):
    c, S = s["case"], s["S"]
    fam = c["family"]
    if fam == "static":
        S.update_material(s["E"])
        S.assemble(gpu.ASM_K_TF32 if c["assembly"] == "tf32" else gpu.ASM_K)
        return S.solve(s["f"], tol=c["tol"], precision=PREC[c["precision"]])[0]
    if fam == "tied":
        for b, E in enumerate(s["E"]):
            S.update_material(E, bucket=b)
        S.assemble()
        return S.solve(s["f"], tol=c["tol"], precision=PREC[c["precision"]])[0]
    if fam == "assemble":
        S.update_coords(s["X"])
        S.update_material(s["E"])
        S.assemble()
        S.assemble_mass()
        return [S.mult_vect(s["x"]), S.mult_vect(s["x"], gpu.ASM_M)]
    if fam == "tangent":
        S.set_displacement(s["u"])
        S.assemble()
        return [S.internal_force(), S.mult_vect(s["x"])]
    if fam == "newton":
        return S.nr_solve(s["q"], c["steps"], 1.0 / c["steps"], tol=1e-10, predictor=c["predictor"],
                          precision=PREC[c["precision"]], lin_tol=1e-10,
                          lin_tol_rel=1e-3 if c["precision"] == "mixed" else 0.0)[0]
    if fam == "newmark":
        return list(S.newmark(s["f"], c["steps"], _NEWMARK_DT, precision=PREC[c["precision"]], tol=1e-10,
                              mass_tol=1e-13)[0])
    S.update_material(s["E"])
    S.assemble()
    return S.solve_batch(s["f"], tol=1e-11)[0]


# --------------------------------------------------------------------- work

def _counts(c):
    """(elements, nodes, nodes per element, Gauss points, stored 3x3 blocks)
    of a box of the case's elements."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    if c.get("kind", "hex8") == "hex8":
        nodes = (nx + 1) * (ny + 1) * (nz + 1)
        return nx * ny * nz, nodes, 8, 8, (3 * nx + 1) * (3 * ny + 1) * (3 * nz + 1)
    v = (nx + 1) * (ny + 1) * (nz + 1)
    e = nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz
    return nx * ny * nz, v + e, 20, 27, 81 * v + 51 * e


def work(case):
    """Each input read once, each result (the assembled blocks among them)
    written once, and the integration's multiply-adds.  A solve's iterations
    are not counted: how much each must move depends on the method."""
    c, fam = case, case["family"]
    if fam == "tied":
        ne8, n8, _, _, b8 = _counts({"kind": "hex8", "nx": c["h8"], "ny": c["h8"], "nz": max(2, c["h8"] // 2)})
        ne20, n20, _, _, b20 = _counts({"kind": "hex20", "nx": c["h20"], "ny": c["h20"], "nz": max(2, c["h20"] // 2)})
        tot_b, tot_f = 72 * (b8 + b20) + 80 * (n8 + n20), 18 * (ne8 * 8 * 36 + ne20 * 27 * 210)
        for p, n in ((2, c["p2"]), (3, c["p3"])):
            k = max(2, n // 4)
            nodes, ne, nn = (n + p) ** 2 * (k + p), n * n * k, (p + 1) ** 3
            tot_b += 72 * nodes * (2 * p + 1) ** 3 + 80 * nodes
            tot_f += 18 * ne * nn * (nn + 1) // 2 * (p + 1) ** 3
        return {"bytes": tot_b, "flops": tot_f}
    if fam == "ensemble":
        ns = np.random.default_rng(c["count"]).integers(c["nmin"], c["nmax"] + 1, size=c["count"])
        got = [_counts({"kind": "hex8", "nx": 2 * int(n), "ny": int(n), "nz": int(n)}) for n in ns]
        ne, nodes, blocks = (sum(g[k] for g in got) for k in (0, 1, 4))
        nn, ng = 8, 8
    else:
        ne, nodes, nn, ng, blocks = _counts(c)
    flops = 18 * ne * ng * nn * (nn + 1) // 2
    bytes_ = 72 * blocks + 24 * nodes + ne * (4 * nn + 16) + 48 * nodes
    if fam == "assemble":
        bytes_ += 72 * blocks + 24 * nodes
    if fam == "newton":
        bytes_ += 24 * nodes * (c["steps"] - 1)
        flops, bytes_ = 3 * flops * c["steps"], bytes_ + 72 * blocks * (c["steps"] - 1)
    if fam == "newmark":
        bytes_ += 72 * blocks + 48 * nodes
    return {"bytes": bytes_, "flops": flops}


# --------------------------------------------------- 64-bit values in torch

def _shapes(kind, ngp):
    """(N [ng, nn], dN/dxi [ng, nn, 3], weights [ng]) on the tensor Gauss grid."""
    nat = torch.tensor(decks.KINDS[kind][1], dtype=torch.float64)
    pts, wts = np.polynomial.legendre.leggauss(ngp)
    g = torch.tensor(np.stack(np.meshgrid(pts, pts, pts, indexing="ij"), -1).reshape(-1, 3))
    w = torch.tensor(np.einsum("i,j,k->ijk", wts, wts, wts).reshape(-1))
    x = g[:, None, :].expand(-1, len(nat), 3).clone().requires_grad_(True)
    if kind == "hex8":
        N = ((1 + x * nat) / 2).prod(-1)
    else:
        t = x * nat
        corner = ((1 + t) / 2).prod(-1) * (t.sum(-1) - 2)
        edge = torch.where(nat == 0, 1 - x * x, (1 + t) / 2).prod(-1)
        N = torch.where((nat == 0).any(-1), edge, corner)
    (dN,) = torch.autograd.grad(N.sum(), x)
    return N.detach(), dN, w


class _Model:
    """Element data of a hex deck on one device in 64 bits."""

    def __init__(self, d, E):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        t = lambda a, k=torch.float64: torch.tensor(a, dtype=k, device=self.dev)  # noqa: E731
        self.conn, self.eq = t(d.conn, torch.int64), t(d.node_eq(), torch.int64)
        self.neq = int(self.eq.max())
        self.X, self.nn = t(d.coords), d.conn.shape[1]
        self.E, self.nu = t(E), t(d.nu)
        self.rho = None if d.rho is None else t(d.rho)
        self.N, self.dN, self.w = (a.to(self.dev) for a in _shapes(d.kind, d.ngp[0]))
        self.dof = self.eq[self.conn].reshape(len(d.conn), -1)  # 0 = no equation

    def chunks(self):
        step = max(1, 16384 * 8 // self.nn)
        return (slice(i, min(i + step, len(self.conn))) for i in range(0, len(self.conn), step))

    def points(self, s):
        """(dN/dx [m, nn, 3], w det J [m]) at each Gauss point of the elements s."""
        X = self.X[self.conn[s]]
        for g in range(len(self.w)):
            J = torch.einsum("ap,eaq->epq", self.dN[g], X)
            yield g, torch.linalg.solve(J, self.dN[g].T.expand(len(X), 3, self.nn)).transpose(1, 2), \
                self.w[g] * torch.linalg.det(J)

    def law(self, s):
        """6x6 isotropic elasticity matrix (engineering shear) of the elements s."""
        E, nu = self.E[s], self.nu[s]
        lam, mu = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
        C = torch.zeros(len(E), 6, 6, dtype=torch.float64, device=self.dev)
        C[:, :3, :3] = lam[:, None, None]
        for k in range(3):
            C[:, k, k] += 2 * mu
            C[:, 3 + k, 3 + k] = mu
        return C

    def strain_rows(self, D, F=None):
        """B [m, 6, 3 nn]: strains of the nodal displacements (of the TL
        variation at deformation gradient F when given)."""
        m = len(D)
        if F is None:
            F = torch.eye(3, dtype=torch.float64, device=self.dev).expand(m, 3, 3)
        B = torch.zeros(m, 6, self.nn, 3, dtype=torch.float64, device=self.dev)
        for k, (i, j) in enumerate([(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]):
            B[:, k] = F[:, None, :, i] * D[:, :, j, None]
            if i != j:
                B[:, k] += F[:, None, :, j] * D[:, :, i, None]
        return B.reshape(m, 6, 3 * self.nn)

    def stiffness(self, u=None):
        """Element matrices; with u (per equation) the TL tangent and the
        element forces too."""
        m, nd = len(self.conn), 3 * self.nn
        K = torch.zeros(m, nd, nd, dtype=torch.float64, device=self.dev)
        G = torch.zeros(m, nd, dtype=torch.float64, device=self.dev)
        ue = None if u is None else self.at(u).reshape(m, self.nn, 3)
        eye = torch.eye(3, dtype=torch.float64, device=self.dev)
        for s in self.chunks():
            C = self.law(s)
            for _, D, c in self.points(s):
                if u is None:
                    B = self.strain_rows(D)
                    K[s] += torch.einsum("e,eki,ekl,elj->eij", c, B, C, B)
                    continue
                F = eye + torch.einsum("eai,eaj->eij", ue[s], D)
                Eg = 0.5 * (F.transpose(1, 2) @ F - eye)
                ev = torch.stack([Eg[:, 0, 0], Eg[:, 1, 1], Eg[:, 2, 2], 2 * Eg[:, 0, 1], 2 * Eg[:, 0, 2],
                                  2 * Eg[:, 1, 2]], 1)
                sv = torch.einsum("ekl,el->ek", C, ev)
                B = self.strain_rows(D, F)
                G[s] += torch.einsum("e,eki,ek->ei", c, B, sv)
                S = torch.stack([sv[:, 0], sv[:, 3], sv[:, 4], sv[:, 3], sv[:, 1], sv[:, 5], sv[:, 4], sv[:, 5],
                                 sv[:, 2]], 1).reshape(-1, 3, 3)
                geo = torch.einsum("e,eai,eij,ebj->eab", c, D, S, D)
                K[s] += torch.einsum("e,eki,ekl,elj->eij", c, B, C, B) + \
                    torch.einsum("eab,ij->eaibj", geo, eye).reshape(-1, nd, nd)
        return K, G

    def mass(self):
        m, nn = len(self.conn), self.nn
        M = torch.zeros(m, nn, nn, dtype=torch.float64, device=self.dev)
        for s in self.chunks():
            for g, _, c in self.points(s):
                M[s] += (c * self.rho[s])[:, None, None] * torch.outer(self.N[g], self.N[g])
        eye = torch.eye(3, dtype=torch.float64, device=self.dev)
        return torch.einsum("eab,ij->eaibj", M, eye).reshape(m, 3 * nn, 3 * nn)

    def at(self, v):
        """Element values of a vector over the equations (0 at supports)."""
        return torch.cat([torch.zeros(1, dtype=torch.float64, device=self.dev), v])[self.dof]

    def gather(self, ve):
        out = torch.zeros(self.neq + 1, dtype=torch.float64, device=self.dev)
        return out.index_add_(0, self.dof.reshape(-1), ve.reshape(-1))[1:]

    def mul(self, Ke, v):
        return self.gather(torch.bmm(Ke, self.at(v)[:, :, None]))

    def solve(self, Ke, f, x=None, tol=3e-15, cap=30000):
        """Jacobi PCG, restarted from the true residual a few times, so that
        the answer is as exact as 64 bits allow."""
        dinv = 1.0 / self.gather(torch.diagonal(Ke, dim1=1, dim2=2))
        x = torch.zeros_like(f) if x is None else x.clone()
        fn = float(f.norm())
        if fn == 0.0:
            return x
        for goal in (1e-12, 1e-3, 1e-2):  # of |f|, then of the residual left
            r = f - self.mul(Ke, x)
            stop = max(goal * (fn if goal < 1e-6 else float(r.norm())), tol * fn)
            z = dinv * r
            p, rz = z.clone(), r @ z
            for it in range(1, cap):
                q = self.mul(Ke, p)
                a = rz / (p @ q)
                x += a * p
                r -= a * q
                if it % 20 == 0 and float(r.norm()) < stop:
                    break
                z = dinv * r
                new = r @ z
                p = z + (new / rz) * p
                rz = new
        return x


def _vec(m, a):
    return torch.tensor(a, dtype=torch.float64, device=m.dev)


def exact(case, seed):
    fam = case["family"]
    if fam == "tied":
        return None  # B-spline solids and multi-point ties: no plain torch form here
    d, a = _inputs(case, seed)
    m = _Model(d, a.get("E", d.E))
    if fam in ("static", "ensemble"):
        return m.solve(m.stiffness()[0], _vec(m, a["f"])).cpu()
    if fam == "assemble":
        x = _vec(m, a["x"])
        return [m.mul(m.stiffness()[0], x).cpu(), m.mul(m.mass(), x).cpu()]
    if fam == "tangent":
        K, G = m.stiffness(_vec(m, a["u"]))
        return [m.gather(G).cpu(), m.mul(K, _vec(m, a["x"])).cpu()]
    if fam == "newton":
        q = _vec(m, a["q"])
        u, steps = torch.zeros_like(q), []
        for k in range(1, case["steps"] + 1):
            f = q * (k / case["steps"])
            for _ in range(30):
                K, G = m.stiffness(u)
                r = f - m.gather(G)
                if float(r.norm()) < 1e-12 * float(f.norm()):
                    break
                u = u + m.solve(K, r, tol=1e-9)
            steps.append(u.cpu())
        return torch.stack(steps)
    # Newmark, average acceleration, from rest
    q, K, M = _vec(m, a["f"]), m.stiffness()[0], m.mass()
    dt, g, b = _NEWMARK_DT, 0.5, 0.25
    u, v = torch.zeros_like(q), torch.zeros_like(q)
    acc = m.solve(M, q)
    Ke = K + M / (b * dt * dt)
    for _ in range(case["steps"]):
        w = u / (b * dt * dt) + v / (b * dt) + (0.5 / b - 1) * acc
        un = m.solve(Ke, q + m.mul(M, w), x=u)
        an = (un - u) / (b * dt * dt) - v / (b * dt) - (0.5 / b - 1) * acc
        v = v + (1 - g) * dt * acc + g * dt * an
        u, acc = un, an
    return [u.cpu(), v.cpu(), acc.cpu()]
