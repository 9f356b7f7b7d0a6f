"""The work that programs have this library do, as cases that can be timed and
checked: batches of Gaussian pairs collocated onto and integrated from periodic
grids, in both precisions, on orthorhombic, multigrid and general cells; forces;
a geometry step; one pair through the drop-in entry; the dense cube cores.

A case's "kind" says which call it is ("batch": collocate and / or integrate of
one task set, "forces": the backward pass, "md": a geometry update and the
collocation after it, "dropin": one pair on host buffers, "core": the dense
contractions).  Inputs are seeded synthetic pairs with the distributions of the
benchmark suite (exponents log-uniform, centres uniform in the cell, blocks and
potentials uniform in [-1, 1], radius from eps = 1e-10).
"""
import ctypes as C
import math

import numpy as np
import torch

from libgpw_gb300 import capi, tasks as T

DEV = "cuda:0"


def _batch(name, op, prec, pairs, lmax, zlo, zhi, cell, n, ny=0, nz=0, levels=1, ortho=True, func=0, tz=-1, kind="batch"):
    c = {"kind": kind, "op": op, "prec": prec, "pairs": pairs, "lmax": lmax, "zlo": zlo, "zhi": zhi, "cell": cell,
         "nx": n, "ny": ny or n, "nz": nz or n, "levels": levels, "ortho": ortho, "func": func, "tz": tz}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a code that calls the reference's single-pair entry, one pair per call on its host grid
        {"name": "dropin_pair", "kind": "dropin", "lmax": 1, "zlo": 0.16, "zhi": 0.5, "cell": 7.56, "nx": 20, "ortho": True,
         "func": 0, "sum_l": False},
        # the prototype's dense contractions, both directions
        {"name": "core_dense", "kind": "core", "nz": 13, "ny": 45, "nx": 29, "L": 7},
        # a small molecule: one SCF step (density to the grid, potential back), plain FP64
        _batch("small_fp64", "both", "fp64", 1000, 2, 0.1, 50.0, 10.0, 64),
        # the same step in mixed precision: launches and latency count
        _batch("small_mixed", "both", "mixed", 1000, 2, 0.1, 50.0, 10.0, 64),
        # kinetic-energy density (meta-GGA) on a ragged grid, FP64
        _batch("tau_fp64", "both", "fp64", 600, 2, 0.1, 50.0, 12.0, 81, 90, 77, func=1),
        # forces and exponent gradients of a medium system
        _batch("forces", "all", "fp64", 2000, 2, 0.1, 50.0, 12.0, 96, kind="forces"),
        # a general cell as a program gets it without tuning, and with the tiles the tuner picks
        _batch("general_mixed", "both", "mixed", 1500, 4, 0.1, 100.0, 15.0, 128, ortho=False),
        _batch("general_tiled", "both", "mixed", 8000, 4, 0.1, 100.0, 15.0, 128, ortho=False, tz=8),
        # three-level multigrid, pairs routed by exponent
        _batch("multigrid_mixed", "both", "mixed", 60000, 3, 0.05, 200.0, 20.0, 180, levels=3),
        # molecular dynamics: new centres, then the density on the new geometry
        _batch("md_step", "collocate", "mixed", 50000, 2, 0.5, 200.0, 20.0, 125, kind="md"),
        # large systems, each direction
        _batch("large_collocate", "collocate", "mixed", 100000, 4, 0.05, 200.0, 30.0, 256),
        _batch("large_integrate", "integrate", "mixed", 100000, 4, 0.05, 200.0, 30.0, 256),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["dropin", "core", "fp64", "fp64", "mixed", "mixed", "mixed", "general", "general", "multigrid",
                       "forces", "md"])
    if kind == "dropin":
        return {"kind": "dropin", "lmax": rng.randint(0, 3), "zlo": 0.08, "zhi": round(_log(rng, 0.2, 2.0), 3),
                "cell": round(rng.uniform(6.0, 14.0), 2), "nx": rng.randint(12, 40), "ortho": rng.random() < 0.7,
                "func": rng.randint(0, 1), "sum_l": rng.random() < 0.5}
    if kind == "core":
        return {"kind": "core", "nz": rng.randint(1, 40), "ny": rng.randint(4, 60), "nx": rng.randint(4, 60),
                "L": rng.randint(1, 9)}
    zlo, zhi = round(_log(rng, 0.05, 0.5), 3), round(_log(rng, 20.0, 200.0), 1)
    lmax = rng.randint(1, 4)
    if kind in ("fp64", "forces"):
        n = rng.randint(40, 110)
        cell = round(n * rng.uniform(0.1, 0.2), 2)
        cap = 2000 if kind == "fp64" else 2500
        c = _batch("", "both", "fp64", 0, min(lmax, 3), max(zlo, 0.1), min(zhi, 100.0), cell, n, n + rng.randint(-5, 5),
                   n + rng.randint(-5, 5), ortho=rng.random() < 0.8, func=rng.choice([0, 0, 1]) if kind == "fp64" else 0)
        if kind == "forces":
            c.update(kind="forces", op="all")
        budget = 4e8
    elif kind == "general":
        n = rng.randint(48, 128)
        c = _batch("", "both", "mixed", 0, lmax, max(zlo, 0.1), min(zhi, 100.0), round(n * rng.uniform(0.11, 0.15), 2), n,
                   ortho=False, tz=rng.choice([-1, 8]))
        cap, budget = 8000, 1.5e9
    elif kind == "multigrid":
        n = 4 * rng.randint(12, 45)
        c = _batch("", rng.choice(["both", "collocate", "integrate"]), "mixed", 0, lmax, zlo, zhi,
                   round(n * rng.uniform(0.1, 0.14), 2), n, levels=3)
        cap, budget = 60000, 8e9
    elif kind == "md":
        n = rng.randint(60, 160)
        c = _batch("", "collocate", "mixed", 0, lmax, 0.5, zhi, round(n * rng.uniform(0.12, 0.18), 2), n, kind="md")
        cap, budget = 50000, 8e9
    else:
        n = int(_log(rng, 40, 256))
        c = _batch("", rng.choice(["both", "collocate", "integrate"]), "mixed", 0, lmax, zlo, zhi,
                   round(n * rng.uniform(0.11, 0.16), 2), n, n + rng.randint(-6, 6), n + rng.randint(-6, 6),
                   func=rng.choice([0, 0, 0, 1]))
        cap, budget = 100000, 16e9
    # cubes of at most a few cells' extent (the broadest product Gaussian has exponent 2 zlo)
    c["zlo"] = max(c["zlo"], round(8.0 / c["cell"] ** 2, 3))
    # as many pairs as keep the points of all cubes under the budget
    h3 = c["cell"] ** 3 / (c["nx"] * c["ny"] * c["nz"])
    vol = 0.0
    for _ in range(64):
        z = _log(rng, c["zlo"], c["zhi"]) + _log(rng, c["zlo"], c["zhi"])
        coarse = 1.0 if c["levels"] == 1 or z > 20.0 else 8.0 if z > 2.0 else 64.0
        vol += 4.19 * (math.log(1e10) / z) ** 1.5 / h3 / coarse / 64
    most = int(min(cap, max(20.0, budget / max(vol, 1.0))))
    c["pairs"] = int(_log(rng, max(10, most // 20), most))
    return c


# ---------------------------------------------------------------------------
# inputs

def _cell(c):
    return float(c["cell"]) if c["ortho"] else T.lattice_15(length=float(c["cell"]))


def _workload(c, seed):
    npts = [(c["nx"], c["ny"], c["nz"])]
    route = None
    if c["levels"] == 3:
        npts += [tuple(max(1, n // f) for n in npts[0]) for f in (2, 4)]
        route = T.multigrid_route
    return T.synthetic("case", c["pairs"], c["lmax"], (c["zlo"], c["zhi"]), _cell(c), npts, seed + 1000, route=route,
                       ortho=c["ortho"], compute_tau=c["func"])


def _room(c):
    """Matrix elements of a buffer that holds the blocks of every pair, whatever their shells."""
    return c["pairs"] * ((c["lmax"] + 1) * (c["lmax"] + 2) // 2) ** 2


def _potentials(wl, seed):
    g = torch.Generator(device=DEV).manual_seed(seed + 77)
    return [torch.rand(T.grid_shape(l), dtype=torch.float64, device=DEV, generator=g).mul_(2.0).sub_(1.0) for l in wl.levels]


def _moved(wl, seed):
    """Centres after a step of about 0.1 bohr, as the device arrays an MD code has."""
    rng = np.random.default_rng(seed + 5)
    da = rng.normal(0.0, 0.05, size=(wl.ntasks, 3))
    db = rng.normal(0.0, 0.05, size=(wl.ntasks, 3))
    return wl.tasks["ra"] + da, wl.tasks["rab"] + db - da


def _dropin_task(c, seed):
    """The argument dictionary of one call of the single-pair entry."""
    rng = np.random.default_rng(seed + 31)
    g = T.make_grid(_cell(c), (c["nx"],) * 3, ortho=c["ortho"])
    la, lb = (int(rng.integers(0, c["lmax"] + 1)) for _ in range(2))
    if c["lmax"] == 1:
        la, lb = 1, 0
    zeta, zetb = np.exp(rng.uniform(math.log(c["zlo"]), math.log(c["zhi"]), size=2))
    cell = np.asarray(g["dh"]) * c["nx"]
    fa, fb = rng.uniform(size=3), rng.uniform(size=3)
    df = fb - fa
    m = T.ncoset(max(la, lb))
    d = {"compute_tau": c["func"], "use_ortho": int(c["ortho"]), "la_max": la, "la_min": 0 if c["sum_l"] else la,
         "lb_max": lb, "lb_min": 0 if c["sum_l"] else lb, "zeta": zeta, "zetb": zetb, "rscale": 1.0, "dh": g["dh"],
         "dh_inv": g["dh_inv"], "ra": fa @ cell, "rab": (df - np.round(df)) @ cell, "npts": g["npts"], "ngrid": g["ngrid"],
         "lb_grid": g["lb_grid"], "periodic": g["periodic"], "lmax": la + lb, "maxco": m, "o1": 0, "o2": 0,
         "radius": float(T.radius_rule(zeta + zetb)), "pab": rng.uniform(-1.0, 1.0, size=(m, m))}
    if c["ortho"]:
        d["lb_cube"], d["ub_cube"], d["sphere_bounds"] = capi.sphere_bounds(d["radius"], d["dh"])
    return d


def prepare(case, seed):
    c = case
    if c["kind"] == "dropin":
        return {"case": c, "task": _dropin_task(c, seed), "grid": np.zeros((c["nx"],) * 3)}
    if c["kind"] == "core":
        g = torch.Generator(device=DEV).manual_seed(seed + 9)
        L, ld = c["L"], max(c["nz"], c["ny"], c["nx"])
        r = lambda *s: torch.rand(s, dtype=torch.float64, device=DEV, generator=g).mul_(2.0).sub_(1.0)  # noqa: E731
        return {"case": c, "co": r(L, L, L), "pol": r(3, L, ld), "V": r(c["nz"], c["ny"], c["nx"]), "ld": ld,
                "length": (C.c_int * 3)(c["nz"], c["ny"], c["nx"]),
                "out": torch.empty(c["nz"], c["ny"], c["nx"], dtype=torch.float64, device=DEV),
                "back": torch.empty(L, L, L, dtype=torch.float64, device=DEV)}
    wl = _workload(c, seed)
    ts = capi.TaskSet.from_workload(capi.Plan(wl.levels), wl)
    if c["tz"] >= 0:
        ts.set_tiles([c["tz"]] * len(wl.levels))
    s = {"case": c, "ts": ts, "pab": torch.from_numpy(wl.pab).to(DEV)}
    z = lambda *n: torch.zeros(n, dtype=torch.float64, device=DEV)  # noqa: E731
    if c["op"] in ("both", "collocate"):
        s["grids"] = [z(*T.grid_shape(l)) for l in wl.levels]
    if c["op"] in ("both", "integrate", "all"):
        s["V"] = _potentials(wl, seed)
        s["hab"] = z(_room(c))
    if c["kind"] == "forces":
        s["grad"] = [z(wl.ntasks, 3), z(wl.ntasks, 3), z(wl.ntasks), z(wl.ntasks)]
    if c["kind"] == "md":
        s["moved"] = [torch.from_numpy(np.ascontiguousarray(x)).to(DEV) for x in _moved(wl, seed)]
    return s


def run(state):
    s, c = state, state["case"]
    if c["kind"] == "dropin":
        s["grid"].fill(0.0)
        capi.collocate_pgf_product_rspace(s["task"], s["grid"])
        return s["grid"]
    if c["kind"] == "core":
        lib, st = capi.lib(), torch.cuda.current_stream().cuda_stream
        capi.check(lib.gpw_collocate_core(s["length"], c["L"], s["co"].data_ptr(), s["pol"].data_ptr(), s["ld"],
                                          s["out"].data_ptr(), st))
        capi.check(lib.gpw_integrate_core(s["length"], c["L"], s["pol"].data_ptr(), s["ld"], s["V"].data_ptr(),
                                          s["back"].data_ptr(), st))
        return s["out"], s["back"]
    ts = s["ts"]
    if c["kind"] == "forces":
        s["hab"].zero_()
        ts.backward(s["pab"], s["V"], s["hab"], *s["grad"])
        return [s["hab"]] + s["grad"]
    out = []
    if c["kind"] == "md":
        ts.update_geometry(*s["moved"])
    if "grids" in s:
        for g in s["grids"]:
            g.zero_()
        ts.collocate(s["pab"], s["grids"], c["prec"])
        out += s["grids"]
    if "V" in s:
        s["hab"].zero_()
        ts.integrate(s["V"], s["hab"], c["prec"])
        out.append(s["hab"])
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    c = case
    if c["kind"] == "core":
        nz, ny, nx, L = c["nz"], c["ny"], c["nx"], c["L"]
        n = nz * ny * nx
        return {"bytes": 8.0 * (2 * n + 2 * L**3 + 2 * 3 * L * max(nz, ny, nx)),
                "flops": 4.0 * (L * n + L * L * nz * ny + L**3 * nz)}
    if c["kind"] == "dropin":
        n = c["nx"] ** 3
        return {"bytes": 16.0 * n, "flops": 2.0 * (2 * c["lmax"] + 1) * n}
    wl = _workload(c, 0)
    t = wl.tasks
    lp = (t["la_max"] + t["lb_max"]).astype(np.float64) + (2 if c["func"] == 1 else 0)
    L = lp + 1
    flops, nbytes = 0.0, 0.0
    ways = {"both": 2, "all": 2}.get(c["op"], 1)
    for l, lv in enumerate(wl.levels):
        m = t["level"] == l
        h = np.abs(np.linalg.det(np.asarray(lv["dh"]))) ** (1.0 / 3.0)
        r = t["radius"][m] / h
        pts, rows, planes = 4.0 / 3.0 * math.pi * r**3, math.pi * r * r, 2.0 * r
        Lm = L[m] + (2 if c["kind"] == "forces" else 0)
        # one multiply-add per power and point, per row and plane for the outer two contractions
        flops += float((2 * Lm * pts + Lm * (Lm + 1) * rows + Lm * (Lm + 1) * (Lm + 2) / 3 * planes).sum())
        nbytes += 8.0 * int(np.prod(lv["ngrid"]))
    pab = 8.0 * wl.pab.size
    return {"bytes": nbytes * (2 if c["op"] == "both" else 1) + pab * ways + 100.0 * wl.ntasks,
            "flops": flops * (2 if c["op"] == "both" else 1)}


# ---------------------------------------------------------------------------
# the same results in plain FP64 torch

def _expand(pa, pb, A, B):
    """E[i][j][k]: (u + pa)^i (u + pb)^j = sum_k E[i][j][k] u^k."""
    E = np.zeros((A + 1, B + 1, A + B + 1))
    E[0, 0, 0] = 1.0

    def times(p, c):
        q = c * p
        q[1:] += p[:-1]
        return q

    for i in range(A + 1):
        if i:
            E[i, 0] = times(E[i - 1, 0], pa)
        for j in range(1, B + 1):
            E[i, j] = times(E[i, j - 1], pb)
    return E


def _shells(lo, hi):
    """(lx, ly, lz) in coset order."""
    return np.array([(lx, l - lx - lz, lz) for l in range(lo, hi + 1) for lx in range(l, -1, -1) for lz in range(l - lx + 1)])


class _Pair:
    """One pair's powers, cube and grid indices, FP64."""

    def __init__(self, t, lv, ra, rab):
        self.t = t
        self.za, self.zb = float(t["zeta"]), float(t["zetb"])
        self.zp = self.za + self.zb
        f = self.zb / self.zp
        self.pref = float(t["rscale"]) * math.exp(-self.za * f * float(rab[0] * rab[0] + rab[1] * rab[1] + rab[2] * rab[2]))
        self.rp = ra + f * rab
        self.pa, self.pb = self.rp - ra, self.rp - (ra + rab)
        self.a = _shells(int(t["la_min"]), int(t["la_max"]))
        self.b = _shells(int(t["lb_min"]), int(t["lb_max"]))
        self.a0, self.b0 = T.ncoset(int(t["la_min"]) - 1), T.ncoset(int(t["lb_min"]) - 1)
        self.E = [_expand(self.pa[d], self.pb[d], int(t["la_max"]) + 2, int(t["lb_max"]) + 2) for d in range(3)]
        dh, inv = np.asarray(lv["dh"]), np.asarray(lv["dh_inv"])
        n = [int(v) for v in lv["npts"]]
        r = float(t["radius"])
        ar = lambda lo, hi: torch.arange(lo, hi + 1, dtype=torch.float64, device=DEV)  # noqa: E731
        if int(lv["ortho"]):
            h = [float(dh[d, d]) for d in range(3)]
            cc = [math.floor(sum(inv[j, d] * self.rp[j] for j in range(3))) for d in range(3)]
            off = [self.rp[d] - cc[d] * h[d] for d in range(3)]
            k = [math.floor(r / h[d]) for d in range(3)]
            g = [ar(-k[d], k[d] + 1) for d in range(3)]
            fold = [torch.where(v <= 0, -v, v - 1) for v in g]
            remk = (r * r - (fold[2] * h[2]) ** 2).clamp(min=0.0)
            jmax = torch.floor(torch.sqrt(remk) / h[1])
            rem = (remk[:, None] - (fold[1] * h[1])[None, :] ** 2).clamp(min=0.0)
            imax = torch.floor(torch.sqrt(rem) / h[0])
            self.mask = (fold[1][None, :, None] <= jmax[:, None, None]) & (fold[0][None, None, :] <= imax[:, :, None])
            self.x = [(g[d] * h[d] - off[d]).view([-1 if d == 2 - i else 1 for i in range(3)]) for d in range(3)]
            self.r2 = sum(x * x for x in self.x)
            idx = [(g[d].long() + cc[d]) % n[d] for d in range(3)]
        else:
            gp = inv.T @ self.rp
            ext = r * np.sqrt((inv**2).sum(axis=0))  # the sphere's half width in index units
            lo, hi = np.floor(gp - ext).astype(int), np.ceil(gp + ext).astype(int)
            i = [ar(int(lo[d]), int(hi[d])) for d in range(3)]
            p = [i[d].view([-1 if d == 2 - q else 1 for q in range(3)]) - float(gp[d]) for d in range(3)]
            self.x = [p[0] * float(dh[0, k]) + p[1] * float(dh[1, k]) + p[2] * float(dh[2, k]) for k in range(3)]
            self.r2 = sum(x * x for x in self.x)
            self.mask = self.r2 <= r * r
            idx = [i[d].long() % n[d] for d in range(3)]
        self.index = ((idx[2][:, None, None] * n[1] + idx[1][None, :, None]) * n[0] + idx[0][None, None, :])
        self.w = torch.where(self.mask, torch.exp(-self.zp * self.r2), torch.zeros((), dtype=torch.float64, device=DEV))

    # one axis' expansion after a derivative: the entries for the pair's own shells
    def plain(self, d):
        return self.E[d]

    def both_d(self, d):  # d phi_a d phi_b
        E, F = self.E[d], np.zeros_like(self.E[d])
        A, B = E.shape[0] - 2, E.shape[1] - 2
        for i in range(A):
            for j in range(B):
                F[i, j] = 4.0 * self.za * self.zb * E[i + 1, j + 1]
                if i:
                    F[i, j] -= 2.0 * self.zb * i * E[i - 1, j + 1]
                if j:
                    F[i, j] -= 2.0 * self.za * j * E[i + 1, j - 1]
                if i and j:
                    F[i, j] += i * j * E[i - 1, j - 1]
        return F

    def centre(self, d, which):  # d / d centre
        E, F = self.E[d], np.zeros_like(self.E[d])
        for i in range(E.shape[0] - 1):
            for j in range(E.shape[1] - 1):
                if which == 0:
                    F[i, j] = 2.0 * self.za * E[i + 1, j] - (i * E[i - 1, j] if i else 0.0)
                else:
                    F[i, j] = 2.0 * self.zb * E[i, j + 1] - (j * E[i, j - 1] if j else 0.0)
        return F

    def square(self, d, which):  # (x - centre)^2 phi
        E, F = self.E[d], np.zeros_like(self.E[d])
        if which == 0:
            F[:-2] = E[2:]
        else:
            F[:, :-2] = E[:, 2:]
        return F

    def weights(self, X):
        """Per axis (nb * na, powers): the expansions of each block element's factor."""
        return [X[d][self.a[None, :, d], self.b[:, None, d]].reshape(len(self.a) * len(self.b), -1) for d in range(3)]

    def terms(self, func):
        if func == 0:
            return [(1.0, [self.plain(d) for d in range(3)])]
        return [(0.5, [self.both_d(d) if d == e else self.plain(d) for d in range(3)]) for e in range(3)]

    def poly(self, block, terms):
        """c[z][y][x] of the product polynomial."""
        c = 0.0
        for f, X in terms:
            x, y, z = self.weights(X)
            zy = (f * block.reshape(-1, 1) * z)[:, :, None] * y[:, None, :]
            c = c + (zy.reshape(len(z), -1).T @ x).reshape(z.shape[1], y.shape[1], x.shape[1])
        return self.pref * c

    def powers(self, d, n):
        p = [torch.ones_like(self.x[d])]
        for _ in range(n - 1):
            p.append(p[-1] * self.x[d])
        return p

    def values(self, c):
        """sum_zyx c x^. y^. z^. exp(-zp r^2) over the cube."""
        n = max([k + 1 for ax in range(3) for k in range(c.shape[ax]) if np.any(np.take(c, k, axis=ax))], default=1)
        c = c[:n, :n, :n]
        if self.x[0].numel() == self.x[0].shape[2]:  # separable
            X, Y, Z = (torch.stack([q.reshape(-1) for q in self.powers(d, n)]) for d in range(3))
            t = torch.from_numpy(np.ascontiguousarray(c)).to(DEV)
            return torch.einsum("zyx,zk,yj,xi->kji", t, Z, Y, X) * self.w
        out = torch.zeros_like(self.w)
        for kz in range(n - 1, -1, -1):
            sy = torch.zeros_like(self.w)
            for ky in range(n - 1 - kz, -1, -1):
                sx = torch.zeros_like(self.w)
                for kx in range(n - 1 - kz - ky, -1, -1):
                    sx.mul_(self.x[0]).add_(float(c[kz, ky, kx]))
                sy.mul_(self.x[1]).add_(sx)
            out.mul_(self.x[2]).add_(sy)
        return out * self.w

    def moments(self, V, n):
        """m[z][y][x] = sum over the cube of V exp(-zp r^2) x^. y^. z^. up to total degree n - 1."""
        v = V.reshape(-1)[self.index] * self.w
        if self.x[0].numel() == self.x[0].shape[2]:
            X, Y, Z = (torch.stack([q.reshape(-1) for q in self.powers(d, n)]) for d in range(3))
            return torch.einsum("kji,zk,yj,xi->zyx", v, Z, Y, X).cpu().numpy()
        m = torch.zeros((n, n, n), dtype=torch.float64, device=DEV)
        vz = v
        for kz in range(n):
            vy = vz
            for ky in range(n - kz):
                vx = vy
                for kx in range(n - kz - ky):
                    m[kz, ky, kx] = vx.sum()
                    vx = vx * self.x[0]
                vy = vy * self.x[1]
            vz = vz * self.x[2]
        return m.cpu().numpy()

    def back(self, m, terms):
        """Matrix elements (nb, na) of the moments m[z][y][x]."""
        n = m.shape[0]
        h = 0.0
        for f, X in terms:
            x, y, z = (np.pad(w[:, :n], ((0, 0), (0, max(0, n - w.shape[1])))) for w in self.weights(X))
            zy = (x @ m.reshape(n * n, n).T).reshape(-1, n, n)
            h = h + f * (((zy * y[:, None, :]).sum(axis=2)) * z).sum(axis=1)
        return self.pref * h.reshape(len(self.b), len(self.a))


def exact(case, seed):
    c = case
    if c["kind"] == "core":
        s = prepare(c, seed)
        P = s["pol"]
        Z, Y, X = P[0][:, :c["nz"]], P[1][:, :c["ny"]], P[2][:, :c["nx"]]
        return (torch.einsum("agb,gz,by,ax->zyx", s["co"], Z, Y, X), torch.einsum("zyx,gz,by,ax->gba", s["V"], Z, Y, X))
    if c["kind"] == "dropin":
        d = _dropin_task(c, seed)
        lv = T.make_grid(_cell(c), (c["nx"],) * 3, ortho=c["ortho"])
        p = _Pair(d, lv, d["ra"], d["rab"])
        block = d["pab"][p.b0:p.b0 + len(p.b), p.a0:p.a0 + len(p.a)]
        g = torch.zeros((c["nx"],) * 3, dtype=torch.float64, device=DEV)
        g.view(-1).index_add_(0, p.index.reshape(-1), p.values(p.poly(block, p.terms(c["func"]))).reshape(-1))
        return g.cpu().numpy()
    if c["pairs"] > (300 if not c["ortho"] else 2100):
        return None
    wl = _workload(c, seed)
    ra, rab = _moved(wl, seed) if c["kind"] == "md" else (wl.tasks["ra"], wl.tasks["rab"])
    grids = [torch.zeros(T.grid_shape(l), dtype=torch.float64, device=DEV) for l in wl.levels]
    V = _potentials(wl, seed)
    hab = np.zeros(_room(c))
    grad = [np.zeros((wl.ntasks, 3)), np.zeros((wl.ntasks, 3)), np.zeros(wl.ntasks), np.zeros(wl.ntasks)]
    for k in range(wl.ntasks):
        t = wl.tasks[k]
        p = _Pair(t, wl.levels[int(t["level"])], ra[k], rab[k])
        o, size = int(t["pab_offset"]), len(p.a) * len(p.b)
        block = wl.pab[o:o + size].reshape(len(p.b), len(p.a))
        terms = p.terms(c["func"])
        if c["op"] in ("both", "collocate"):
            v = p.values(p.poly(block, terms))
            grids[int(t["level"])].view(-1).index_add_(0, p.index.reshape(-1), v.reshape(-1))
        if c["op"] in ("both", "integrate", "all"):
            lp = int(t["la_max"]) + int(t["lb_max"])
            m = p.moments(V[int(t["level"])], lp + 1 + (2 if c["func"] or c["kind"] == "forces" else 0))
            hab[o:o + size] = p.back(m, terms).reshape(-1)
        if c["kind"] == "forces":
            dot = lambda X: float((p.back(m, [(1.0, X)]) * block).sum())  # noqa: E731
            for d in range(3):
                for q in (0, 1):
                    grad[q][k, d] = dot([p.centre(e, q) if e == d else p.plain(e) for e in range(3)])
                    grad[2 + q][k] -= dot([p.square(e, q) if e == d else p.plain(e) for e in range(3)])
    if c["kind"] == "forces":
        return [hab] + grad
    return (grids if c["op"] in ("both", "collocate") else []) + ([hab] if c["op"] in ("both", "integrate") else [])
