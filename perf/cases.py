"""The calls whose time counts: matvecs in every arithmetic, a time step's
update, velocity fields and the two solves, each through the package's public
entry points (Context of rbc3d_gb300), from three coarse cells to the
2048-cell box.

A case is a dict:
  kind   "matvec"  Context.matvec on the cells' own points, inputs resident;
         "step"    what a time step calls: set_cells_x, set_cell_density_x, matvec;
         "field"   calc_velocity_field at scattered points of the box;
         "cell"    solve_rbc_vel (cell velocity GMRES, spherical-harmonic unknowns);
         "wall"    no_slip_wall (wall density GMRES) in a periodic tube
  prec   "FP64", "FP32C", "FP32D" or "FP32M" (the library's four arithmetics)
  ncell, nlat, nlon    cells and the grid of each
  nb     PME mesh nodes per edge of the box (per tube diameter for "wall")
  dl     double layer beside the single layer
  types  1, or 2: cells of two viscosity ratios
  npoint "field": number of points;  nz  "wall": rings of 48 vertices
"""
import math
from types import SimpleNamespace

import numpy as np
import torch

import rbc3d_gb300 as R
from rbc3d_gb300 import geometry as G

PREC = {"FP64": R.FP64, "FP32C": R.FP32C, "FP32D": R.FP32D, "FP32M": R.FP32M}
C = 1.0 / (4.0 * math.pi)
EPS, RC, ORDER, DEGREE = 1e-6, 3.0, 6, 12
SPACING = 6.3  # box edge per cube root of the cell count: 256 cells in a cube of 40
TUBE_R, TUBE_BOX, TUBE_H = 8.0, 16.5, 0.25


def _case(kind, prec, ncell, nb, nlat=25, nlon=50, dl=True, types=1, npoint=0, nz=0, name=None):
    c = dict(kind=kind, prec=prec, ncell=ncell, nb=nb, nlat=nlat, nlon=nlon, dl=dl, types=types, npoint=npoint, nz=nz)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a first try-out of a set-up: three coarse cells, single layer, the reference's arithmetic
        _case("matvec", "FP64", 3, 32, 12, 24, dl=False, name="matvec fp64 3 coarse SL"),
        # a few cells at full resolution: one call's latency in the default arithmetic
        _case("matvec", "FP32D", 8, 64, name="matvec fp32d 8"),
        # the reference's arithmetic at the size of a tube's cell suspension
        _case("matvec", "FP64", 64, 80, name="matvec fp64 64"),
        # the 256-cell suspension in the three FP32 arithmetics
        _case("matvec", "FP32D", 256, 128, name="matvec fp32d 256"),
        _case("matvec", "FP32C", 256, 128, name="matvec fp32c 256"),
        _case("matvec", "FP32M", 256, 128, name="matvec fp32m 256"),
        # one update of a time step: new positions and densities, then the sums
        _case("step", "FP32D", 256, 128, name="step fp32d 256"),
        # the largest suspension
        _case("matvec", "FP32D", 2048, 256, name="matvec fp32d 2048"),
        # another grid, an odd cell count, cells of two viscosity ratios
        _case("matvec", "FP32D", 97, 90, 24, 48, types=2, name="matvec fp32d 97 of two kinds"),
        # a velocity field for output: points all over the box, on no surface
        _case("field", "FP32D", 64, 80, npoint=20011, name="field fp32d 20011 points"),
        # the cells' surface velocities, mixed precision to the reference's 1e-11
        _case("cell", "FP32D", 61, 80, name="cell solve fp32d 61"),
        # the wall's no-slip density in a short tube, the reference's arithmetic
        _case("wall", "FP64", 16, 96, nz=48, name="wall solve fp64"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh(ncell):
    """An even PME mesh near the suspensions' 3.2 nodes per unit length."""
    return max(32, 2 * int(round(1.6 * SPACING * ncell ** (1 / 3))))


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "matvec", "matvec", "step", "step", "field", "cell", "wall"])
    nlat, nlon = rng.choice([(12, 24), (14, 28), (24, 48), (25, 50), (25, 50), (36, 72)])
    full = 1250.0 / (nlat * nlon)  # cells of the 25 x 50 grid's cost, by points
    dl = rng.random() < 0.75
    types = rng.choice([1, 1, 2]) if dl else 1
    if kind in ("matvec", "step"):
        prec = rng.choice(["FP64", "FP32C", "FP32D", "FP32D", "FP32M"])
        most = {"FP64": 80, "FP32C": 300, "FP32D": 1400, "FP32M": 1400}[prec]
        n = _log(rng, 3, max(4, most * full ** (2 if full < 1 else 1)))
        return _case(kind, prec, n, _mesh(n), nlat, nlon, dl, types)
    if kind == "field":
        n = _log(rng, 3, 200)
        return _case(kind, rng.choice(["FP64", "FP32D"]), n, _mesh(n), 25, 50, dl, types, npoint=_log(rng, 500, 40000))
    if kind == "cell":
        n = _log(rng, 3, 50)
        return _case(kind, rng.choice(["FP32D", "FP32M"]), n, _mesh(n), 25, 50, True, rng.choice([1, 2]))
    return _case(kind, rng.choice(["FP64", "FP32M"]), rng.randint(5, 20), 96, 25, 50, False, 1, nz=rng.choice([40, 44, 48, 56]))


# ---------------------------------------------------------------------------
def _params(case):
    vr = [5.0, 1.0][: case["types"]] if case["dl"] else [1.0]
    if case["kind"] == "wall":
        Lz = TUBE_H * case["nz"]
        Lb, Nb = [TUBE_BOX, TUBE_BOX, Lz], [case["nb"], case["nb"], 2 * int(math.ceil(2.65 * Lz))]
    else:
        Lb, Nb = [max(9.05, SPACING * case["ncell"] ** (1 / 3))] * 3, [case["nb"]] * 3
    return dict(Lb=Lb, alpha=G.alpha_for_cutoff(RC, EPS), rc=RC, eps=EPS, Nb=Nb, P=ORDER, nlat=case["nlat"],
                nlon=case["nlon"], ncelltypes=len(vr), viscRat=vr, vBkg=[0.0, 0.0, 8.0 if case["kind"] == "wall" else 0.0])


def _inputs(case, seed):
    """Biconcave cells at random places and angles (centres at least 2.6
    apart), densities of degree <= 6 with N(0, l^-2) coefficients."""
    rng = np.random.default_rng(seed)
    prm = _params(case)
    n, nlat, nlon = case["ncell"], case["nlat"], case["nlon"]
    th, phi, w = G.gauss_grid(nlat, nlon)
    inside = None
    if case["kind"] == "wall":
        inside = lambda c: (c[0] - TUBE_BOX / 2) ** 2 + (c[1] - TUBE_BOX / 2) ** 2 < 6.3 ** 2  # noqa: E731
    centres = G.place_cells(rng, n, prm["Lb"], 2.6, inside)
    rot = np.stack([G.random_rotation(rng) for _ in range(n)])
    shape = G.biconcave_surface(th, phi, np.eye(3), np.zeros(3))[0]  # (nlat, nlon, 3)
    pts = shape.transpose(1, 0, 2).reshape(nlon * nlat, 3)           # point order: ilon * nlat + ilat
    x = np.einsum("cij,pj->icp", rot, pts) + centres.T[:, :, None]
    modes = [(l, m) for l in range(1, 7) for m in range(-l, l + 1)]
    Y = np.stack([G.sh_eval({k: 1.0}, th, phi).T.reshape(-1) for k in modes])
    sd = np.array([1.0 / l for l, _ in modes])
    f, g = (np.einsum("kcm,mp->kcp", rng.normal(size=(3, n, len(modes))) * sd, Y) for _ in range(2))
    pack = lambda a: np.ascontiguousarray(a.reshape(3, -1))  # noqa: E731
    celltype = (np.arange(n) % case["types"]).astype(np.int32)
    s = SimpleNamespace(prm=prm, th=th, phi=phi, w=w, ncell=n, nlat=nlat, nlon=nlon, celltype=celltype, x=pack(x),
                        f=pack(f), g=pack(g))
    if case["npoint"]:
        s.points = rng.uniform(size=(3, case["npoint"])) * np.array(prm["Lb"])[:, None]
    return s


def _pinned(a):
    """A page-locked copy, as a program that calls every step keeps its arrays."""
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    t.numpy()[...] = a
    return t.numpy()


def _update(s):
    s.ctx.set_cells_x(s.cells, DEGREE)
    s.ctx.set_cell_density_x(DEGREE, f=s.cells.f, g=s.cells.g if s.case["dl"] and s.case["kind"] != "cell" else None)


def prepare(case, seed):
    cells = _inputs(case, seed)
    for k in ("x", "f", "g"):
        setattr(cells, k, _pinned(getattr(cells, k)))
    s = SimpleNamespace(case=case, cells=cells, ctx=R.context(cells.prm), v=_pinned(np.zeros_like(cells.x)))
    if case["kind"] == "wall":
        s.wall = G.make_tube(TUBE_R, TUBE_H * case["nz"], 48, case["nz"], (TUBE_BOX / 2, TUBE_BOX / 2))
        s.zero = np.zeros_like(s.wall.x)
        s.ctx.set_walls(s.wall)
        s.ctx.prepare_sing_int_on_wall()
    _update(s)
    if case["kind"] == "field":
        s.ctx.set_raw_targets(cells.points)
    return s


def run(s):
    case, ctx, prec = s.case, s.ctx, PREC[s.case["prec"]]
    if case["kind"] == "field":
        return ctx.calc_velocity_field(R.TLIST_RAW, prec)
    if case["kind"] == "cell":
        sol, v, _, _ = ctx.solve_rbc_vel(DEGREE, rtol=1e-11, prec=prec)
        return {"sol": sol, "v": v}
    if case["kind"] == "wall":
        ctx.set_wall_density(s.zero)
        ctx.no_slip_wall(1e-8, 600, 300, prec)
        return ctx.get_wall_density(s.wall.nvert)
    if case["kind"] == "step":
        _update(s)
    s.v[...] = 0.0  # matvec adds to the caller's accumulator
    return ctx.matvec(R.TLIST_RBC, C, C if case["dl"] else 0.0, R.TERM_ALL, prec, v=s.v)


def work(case):
    """Positions and densities once in, velocities once out; the flops of the
    formulas: pairs within the cut-off, the own-cell patch quadrature, the
    mesh (spreading, transforms, gather); for a solve, of one operator pass
    for each tenth power that its residual falls by."""
    nv = case["nlat"] * case["nlon"]
    n = case["ncell"] * nv
    prm = _params(case)
    grid = float(np.prod(prm["Nb"]))
    comp = 12 if case["dl"] else 3
    mesh = n * 216 * 2 * (comp + 3) + grid * (comp + 3) * 2.5 * math.log2(grid)
    if case["kind"] == "wall":
        el, nvert = 2 * 48 * case["nz"], 48 * (case["nz"] + 1)
        mesh = (el + nvert) * 216 * 2 * 3 + grid * 6 * 2.5 * math.log2(grid)
        return {"bytes": 8.0 * (6 * n + 9 * nvert), "flops": 8 * mesh + 4e3 * nvert}
    nrad = 2 * int(round(math.pi / math.sqrt(case["nlat"]) / (math.pi / case["nlat"])))
    near = n / float(np.prod(prm["Lb"])) * 4 / 3 * math.pi * RC ** 3  # other cells' points within the cut-off
    per_pair, per_patch = (66, 550) if case["dl"] else (39, 294)
    if case["kind"] == "field":
        m = case["npoint"]
        return {"bytes": 8.0 * ((9 if case["dl"] else 6) * n + 6 * m), "flops": m * near * per_pair + mesh}
    one = n * ((near + nv) * per_pair + 2 * nrad * nrad * per_patch) + mesh
    passes = 12 if case["kind"] == "cell" else 1
    return {"bytes": 8.0 * (12 if case["dl"] else 9) * n, "flops": passes * one}


# ---------------------------------------------------------------------------
# The same sums in plain 64-bit torch: the reference's definitions, every
# pair, projection and transform written out.
NTAB = 8192


def _quad(n, a, b):
    x, w = np.polynomial.legendre.leggauss(n)
    return 0.5 * (b + a) + 0.5 * (b - a) * x, 0.5 * (b - a) * w


def _legendre(L, th):
    """P(row, m, n) of unit norm on [-1, 1], and dP/dtheta."""
    x, s = np.cos(th), np.sin(th)
    P, D = np.zeros((th.size, L, L)), np.zeros((th.size, L, L))
    for m in range(L):
        P[:, m, m] = math.sqrt(0.5) if m == 0 else P[:, m - 1, m - 1] * math.sqrt((2 * m + 1) / (2 * m)) * s
        for n in range(m + 1, L):
            a = math.sqrt((4.0 * n * n - 1) / (n * n - m * m))
            b = math.sqrt(((n - 1.0) ** 2 - m * m) / (4.0 * (n - 1.0) ** 2 - 1)) if n > m + 1 else 0.0
            P[:, m, n] = a * (x * P[:, m, n - 1] - b * P[:, m, n - 2])
    for m in range(L):
        for n in range(m, L):
            up = math.sqrt((n - m) * (n + m + 1.0)) * P[:, m + 1, n] if m + 1 <= n else 0.0
            down = math.sqrt((n + m) * (n - m + 1.0)) * P[:, m - 1, n] if m else 0.0
            D[:, m, n] = 0.5 * (down - up) if m else -up
    return P, D


class _Exact:
    def __init__(self, case, seed):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        s = _inputs(case, seed)
        self.case, self.s, self.prm = case, s, s.prm
        self.n, self.nlat, self.nlon, self.nv = s.ncell, s.nlat, s.nlon, s.nlat * s.nlon
        self.L = self.t(s.prm["Lb"])
        vr = np.array(s.prm["viscRat"])[s.celltype]
        self.A, self.B = self.t(1 + vr), self.t(1 - vr)
        self.field = lambda a: self.t(a).reshape(3, self.n, self.nlon, self.nlat).permute(1, 3, 2, 0)  # (cell, lat, lon, 3)
        self.th, self.phi, self.w = self.t(s.th), self.t(s.phi), self.t(s.w)
        self.radius = math.pi / math.sqrt(self.nlat)
        self.c1, self.c2 = C, C if case["dl"] else 0.0
        self.tables()
        self.geometry()

    def t(self, a):
        return torch.as_tensor(np.asarray(a, dtype=np.float64), device=self.dev)

    # -- tables of the kernels and of the mask, linear between their nodes
    def tables(self):
        a, rc = self.prm["alpha"], RC
        r = np.sqrt(math.pi / a) * np.arange(NTAB + 1) * rc / NTAB
        erfc = np.array([math.erfc(v) for v in r])
        ex = np.exp(-r * r)
        self.tab = self.t([erfc, 2 / math.sqrt(a) * ex,
                           -8 / math.sqrt(math.pi) * (ex * (1.5 * r + r ** 3) + 0.75 * math.sqrt(math.pi) * erfc)])
        u = np.arange(NTAB + 1) / NTAB
        with np.errstate(divide="ignore", over="ignore"):
            m = np.exp(2 * np.exp(-1 / np.maximum(u, 1e-300)) / np.where(u < 1, u - 1, -1e-300))
        self.mtab = self.t(np.where(u < 0.01, 1.0, np.where(u > 0.99, 0.0, m)))

    def mask(self, x):
        s = x.abs() * NTAB
        i = s.floor().clamp(max=NTAB - 1).long()
        return torch.where(s < NTAB, self.mtab[i] * (i + 1 - s) + self.mtab[i + 1] * (s - i), torch.zeros_like(s))

    def kernels(self, d, F, Gd, N, wt):
        """sum over the last point axis of wt (c1 SL F + c2 DL (Gd, N)) at offsets d (..., q, 3)."""
        r2 = (d * d).sum(-1)
        r = r2.sqrt()
        ok = r >= 1e-3 * math.sqrt(self.prm["alpha"] / math.pi)
        r = torch.where(ok, r, torch.ones_like(r))
        s = r * (NTAB / RC)
        ok &= s < NTAB
        i = s.floor().clamp(max=NTAB - 1).long()
        T = lambda k: self.tab[k][i] * (i + 1 - s) + self.tab[k][i + 1] * (s - i)  # noqa: E731
        wt = torch.where(ok, wt, torch.zeros_like(wt))
        t1, t2 = T(0), T(1)
        EA, EB = (t1 / r + t2) / (r * r), t1 / r - t2
        v = (self.c1 * wt * EA * (d * F).sum(-1))[..., None] * d + (self.c1 * wt * EB)[..., None] * F
        if self.c2:
            v = v + (self.c2 * wt * T(2) / r ** 5 * (d * Gd).sum(-1) * (d * N).sum(-1))[..., None] * d
        return v.sum(-2)

    # -- geometry of degree < nlat, filtered spline tables of degree < DEGREE
    def geometry(self):
        s, nlat, nlon = self.s, self.nlat, self.nlon
        m = np.arange(nlat)
        cs, sn = np.cos(np.outer(m, s.phi)), np.sin(np.outer(m, s.phi))
        wf = s.w / math.pi
        P, D = _legendre(nlat, s.th)
        eq = np.arange(nlat + 1) * (math.pi / nlat)
        PE = _legendre(DEGREE, eq)[0]
        half = np.where(m == 0, 0.5, 1.0)
        P, D, PE, cs, sn, wf, half, mm = (self.t(v) for v in (P, D, PE, cs, sn, wf, half, m))

        def anal(v):  # (cell, lat, lon, k) -> cosine and sine parts (cell, m, n, k)
            return tuple(torch.einsum("imn,i,cijk,mj->cmnk", P, wf, v, q) for q in (cs, sn))

        X = self.field(s.x)
        mean = X.mean((1, 2), keepdim=True)
        a, b = anal(X - mean)
        syn = lambda Q, f, g: torch.einsum("m,imn,cmnk,mj->cijk", half, Q, a, f) + torch.einsum("m,imn,cmnk,mj->cijk", half, Q, b, g)  # noqa: E731
        xt, xp = syn(D, cs, sn), syn(P, -mm[:, None] * sn, mm[:, None] * cs)
        nrm = torch.cross(xt, xp, dim=-1)
        size = nrm.norm(dim=-1, keepdim=True)
        self.N = nrm / size
        self.J = size[..., 0] / self.th.sin()[:, None]
        self.X, self.F, self.G = X, self.field(s.f), self.field(s.g)
        dS = self.J * self.w[:, None]
        self.area = dS.sum((1, 2))
        self.size = (self.area / nlat ** 2).sqrt()
        self.dF, self.dG = self.F * dS[..., None], self.G * dS[..., None] * self.B[:, None, None, None]

        def spline(v):  # filtered, on the doubled meridian grid: (cell, 2 nlat, nlon, k, 4)
            k, c0 = DEGREE, v.mean((1, 2), keepdim=True)
            a, b = (q[:, :k, :k] for q in anal(v - c0))
            e = torch.einsum("m,imn,cmnk,mj->cijk", half[:k], PE, a, cs[:k]) + torch.einsum("m,imn,cmnk,mj->cijk", half[:k], PE, b, sn[:k])
            e = e + c0
            u = torch.cat([e[:, :-1], torch.roll(e[:, 1:].flip(1), -(nlon // 2), 2)], 1)
            return torch.stack([u, self.diff(u, 1), self.diff(u, 2), self.diff(self.diff(u, 1), 2)], -1)

        J1 = self.J[..., None]
        self.spl = {"x": spline(X), "n": spline(self.N), "j": spline(J1), "f": spline(self.F * J1), "g": spline(self.G * J1)}
        # one table for an interpolation of all: x, f, g, n
        self.all = torch.cat([self.spl[k] for k in "xfgn"], 3).flatten(1, 2)  # (cell, node, 12, 4)
        self.pts = lambda v: v.transpose(1, 2).reshape(self.n, self.nv, -1)   # (cell, point, k)

    @staticmethod
    def diff(u, axis):
        n = u.shape[axis]
        k = torch.arange(n // 2 + 1, dtype=torch.float64, device=u.device)
        k[-1] = 0
        shape = [1] * u.dim()
        shape[axis] = k.numel()
        return torch.fft.irfft(torch.fft.rfft(u, dim=axis) * (1j * k).reshape(shape), n=n, dim=axis)

    def interp(self, tab, cell, th, phi):
        """Bicubic Hermite values of tab (cell, node, k, 4) at (th, phi) of `cell` (broadcast)."""
        m, n = 2 * self.nlat, self.nlon
        hx, hy = 2 * math.pi / m, 2 * math.pi / n
        x, y = th / hx, phi / hy
        i, j = x.floor(), y.floor()
        s, t = x - i, y - j
        i, j = i.long(), j.long()
        one = lambda q, h: ((1 + q * q * (2 * q - 3), h * q * (1 + q * (q - 2))), (q * q * (3 - 2 * q), h * q * q * (q - 1)))  # noqa: E731
        v = 0
        for a, (cu, cd) in enumerate(one(s, hx)):
            for b, (eu, ed) in enumerate(one(t, hy)):
                node = ((i + a) % m) * n + (j + b) % n
                v = v + torch.einsum("...kd,...d->...k", tab[cell, node], torch.stack([cu * eu, cd * eu, cu * ed, cd * ed], -1))
        return v

    def patch(self, th0, phi0, thL, phL):
        """The point at polar coordinates (thL, phL) about the pole (th0, phi0)."""
        x, y, z = thL.sin() * phL.cos(), thL.sin() * phL.sin(), thL.cos()
        u, v = th0.cos() * x + th0.sin() * z, th0.cos() * z - th0.sin() * x
        p = torch.atan2(y, u) + phi0
        return v.clamp(-1, 1).acos(), p - (p / (2 * math.pi)).floor() * 2 * math.pi

    def image(self, d):
        return d - (d / self.L).round() * self.L

    def sphere_dist(self, t0, p0, t1, p1):
        return ((t0 - t1).cos() - t0.sin() * t1.sin() * (1 - (p0 - p1).cos())).clamp(-1, 1).acos()

    # -- the sums
    def velocity(self, x, A, own):
        """At points x (N, 3) with coefficients A; own: they are the cells' points in order."""
        v = torch.zeros_like(x)
        X, F, Gd, N = (self.pts(q) for q in (self.X, self.dF, self.dG, self.N))
        grid = [self.pts(q.expand(1, self.nlat, self.nlon)[..., None].expand(self.n, -1, -1, -1))[0, :, 0] for q in (self.th[:, None], self.phi[None])]
        items = []
        for c in range(self.n):
            mid = X[c].mean(0)
            reach = (X[c] - mid).norm(dim=-1).max() + RC
            at = (self.image(x - mid).norm(dim=-1) <= reach).nonzero()[:, 0]
            for q in at.split(6000):
                d = self.image(X[c][None] - x[q, None])
                r = d.norm(dim=-1)
                wt = (r <= RC).double()
                if own:
                    same = (q // self.nv == c).nonzero()[:, 0]
                    if same.numel():
                        p = q[same] % self.nv
                        wt[same] *= 1 - self.mask(self.sphere_dist(grid[0][p, None], grid[1][p, None], grid[0][None], grid[1][None]) / self.radius)
                v[q] += self.kernels(d, F[c][None], Gd[c][None], N[c][None], wt)
                r, k = r.min(1)
                r = torch.where(q // self.nv == c, RC + 1.0, r) if own else r
                e = (r <= RC).nonzero()[:, 0]
                items.append((q[e], torch.full_like(e, c), k[e]))
        if own:
            self.own_patch(v)
        self.near(v, x, *(torch.cat(q) for q in zip(*items)))
        if self.c2:
            total = (self.pts(self.X) * (Gd * N).sum(-1, keepdim=True)).sum((0, 1))
            v += self.c2 * (-8 * math.pi / float(self.L.prod())) * total
        self.mesh(v, x)
        return v / A[:, None]

    def rule(self, radius, nrad, nazm):
        thL, pw = _quad(nrad, 0.0, radius)
        thL, pw = self.t(thL), self.t(pw)
        pw = pw * thL.sin() * (2 * math.pi / nazm) * self.mask(thL / radius)
        return thL, pw, torch.arange(nazm, dtype=torch.float64, device=self.dev) * (2 * math.pi / nazm)

    def own_patch(self, v):
        nrad = 2 * round(self.radius / (math.pi / self.nlat))
        thL, pw, phL = self.rule(self.radius, nrad, 2 * nrad)
        cells = torch.arange(self.n, device=self.dev)
        for i in range(self.nlat):
            for c in cells.split(max(1, 2000000 // (self.nlon * nrad * 2 * nrad))):
                th, ph = self.patch(self.th[i], self.phi[:, None, None], thL[None, :, None], phL[None, None])
                th = th.expand(ph.shape).flatten(1)
                val = self.interp(self.all, c[:, None, None], th[None], ph.flatten(1)[None])
                x0 = self.interp(self.all, c[:, None], self.th[i].expand(1, self.nlon), self.phi[None])[..., :3]
                d = val[..., :3] - x0[:, :, None]
                wt = pw[:, None].expand(nrad, 2 * nrad).reshape(-1) * (d.norm(dim=-1) < RC)
                dv = self.kernels(d, val[..., 3:6], val[..., 6:9] * self.B[c, None, None, None], val[..., 9:], wt)
                at = c[:, None] * self.nv + torch.arange(self.nlon, device=self.dev) * self.nlat + i
                v[at] += dv

    def near(self, v, x, q, c, k):
        """Projection of the points onto the cells near them, and the correction of those within two mesh sizes."""
        for q, c, k in zip(q.split(40000), c.split(40000), k.split(40000)):
            X, ilat, ilon = self.pts(self.X)[c, k], k % self.nlat, k // self.nlat
            xt = X + self.image(x[q] - X)
            th, ph, x0 = self.project(c, self.th[ilat], self.phi[ilon], xt)
            n0 = self.interp(self.all, c, th, ph)[..., 9:]
            dist = (n0 * (xt - x0)).sum(-1)
            e = (dist <= 2 * self.size[c]).nonzero()[:, 0]
            q, c, xt, th, ph, x0, n0, dist = (a[e] for a in (q, c, xt, th, ph, x0, n0, dist))
            if not e.numel():
                continue
            dv = -self.subtract(c, xt, th, ph)
            lim = (0.01 * self.radius * (self.area[c] / (4 * math.pi)).sqrt()).copysign(dist)
            far = dist.abs() >= lim.abs()
            a = self.readd(c, torch.where(far[:, None], xt, x0 + lim[:, None] * n0), x0, th, ph)
            b = self.readd(c, x0, x0, th, ph)
            if self.c2:
                g0 = self.interp(self.all, c, th, ph)[..., 6:9] / self.interp(self.spl["j"].flatten(1, 2), c, th, ph)
                b = b + (self.c2 * self.B[c] * 4 * math.pi * torch.where(dist > 0, 1.0, -1.0))[:, None] * g0
            dv = dv + torch.where(far[:, None], a, b + (dist / lim)[:, None] * (a - b))
            v.index_add_(0, q, dv)

    def project(self, c, th, ph, xt):
        h = max(math.pi / self.nlat, 2 * math.pi / self.nlon)
        pos = self.spl["x"].flatten(1, 2)
        x0 = self.interp(pos, c, th, ph)
        live = torch.ones_like(th, dtype=torch.bool)
        k = torch.arange(16, device=self.dev)
        for _ in range(3):
            thL, phL = (k % 2 + 1) * h / 2, (k // 2).double() * (2 * math.pi / 8)
            tp, pp = self.patch(th[:, None], ph[:, None], thL, phL)
            tp, pp = torch.cat([tp, th[:, None]], 1), torch.cat([pp, ph[:, None]], 1)
            d2 = ((self.interp(pos, c[:, None], tp, pp) - xt[:, None]) ** 2).sum(-1)
            z = torch.zeros(1, dtype=torch.float64, device=self.dev)
            px, py = torch.cat([thL * phL.cos(), z]), torch.cat([thL * phL.sin(), z])
            U = torch.stack([torch.ones_like(px), px, py, px * px, px * py, py * py], 1)
            b = torch.linalg.solve(U.T @ U, (d2 @ U).T).T
            det = 4 * b[:, 3] * b[:, 5] - b[:, 4] ** 2
            ok = det > 0
            det = torch.where(ok, det, torch.ones_like(det))
            mx = torch.where(ok, (b[:, 4] * b[:, 2] - 2 * b[:, 5] * b[:, 1]) / det, 0.0)
            my = torch.where(ok, (b[:, 4] * b[:, 1] - 2 * b[:, 3] * b[:, 2]) / det, 0.0)
            tm, pm = self.patch(th, ph, (mx * mx + my * my).sqrt(), torch.atan2(my, mx))
            xm = self.interp(pos, c, tm, pm)
            live = live & (((xm - xt) ** 2).sum(-1) <= d2[:, 16])
            th, ph, x0 = torch.where(live, tm, th), torch.where(live, pm, ph), torch.where(live[:, None], xm, x0)
            h = 0.5 * h
        return th, ph, x0

    def subtract(self, c, xt, th, ph):
        """The mesh points' masked sums within the patch about the projection."""
        X, F, Gd, N = (self.pts(q) for q in (self.X, self.dF, self.dG, self.N))
        g1, g2 = self.th.repeat(self.nlon), self.phi.repeat_interleave(self.nlat)
        out = torch.empty_like(xt)
        for e in torch.arange(c.numel(), device=self.dev).split(500):
            k = c[e]
            m = self.mask(self.sphere_dist(th[e, None], ph[e, None], g1, g2) / self.radius)
            d = X[k] - xt[e, None]
            out[e] = self.kernels(d, F[k], Gd[k], N[k], m * (d.norm(dim=-1) <= RC))
        return out

    def readd(self, c, xi, x0, th0, ph0):
        """The patch about the projection with the sinh-mapped radial rule (16 x 32 points)."""
        out = torch.empty_like(xi)
        g, w = (self.t(q) for q in _quad(16, -1.0, 1.0))
        x1, w1 = (self.t(q) for q in _quad(16, 0.0, self.radius))
        phL = torch.arange(32, dtype=torch.float64, device=self.dev) * (2 * math.pi / 32)
        xl = 0.5 * self.radius
        for e in torch.arange(c.numel(), device=self.dev).split(400):
            d = (xi[e] - x0[e]).norm(dim=-1)
            b = (d * (self.radius / (self.radius * (self.area[c[e]] / (4 * math.pi)).sqrt())) * xl)[:, None]
            at = b > 0
            bb = torch.where(at, b, torch.ones_like(b))
            u1, u2 = torch.zeros_like(bb), (2 / bb).asinh()  # the interval's ends: 0 and 2 half-lengths from the pole
            mu, eta = 0.5 * (u1 + u2), 0.5 * (u1 - u2)
            thL = torch.where(at, xl + xl * (-1 + bb * (mu * g - eta).sinh()), x1)
            wt = torch.where(at, xl * w * bb * mu * (mu * g - eta).cosh(), w1)
            wt = wt * thL.sin() * (2 * math.pi / 32) * self.mask(thL / self.radius)
            th, ph = self.patch(th0[e, None, None], ph0[e, None, None], thL[:, :, None], phL)
            val = self.interp(self.all, c[e, None, None], th, ph).flatten(1, 2)
            dd = val[..., :3] - xi[e, None]
            wt = wt[:, :, None].expand(-1, -1, 32).flatten(1) * (dd.norm(dim=-1) <= RC)
            out[e] = self.kernels(dd, val[..., 3:6], val[..., 6:9] * self.B[c[e], None, None], val[..., 9:], wt)
        return out

    # -- mesh part
    def bspline(self, x):
        """Lowest node and the weights (N, 3, P) of points x."""
        Nb = self.t(self.prm["Nb"])
        xc = x * (Nb / self.L)
        lo = xc.floor() - (ORDER - 1)
        u = [lo - (xc - ORDER) + j for j in range(ORDER)]
        w = [torch.ones_like(xc)] + [torch.zeros_like(xc)] * (ORDER - 1)
        for p in range(2, ORDER + 1):
            w = [u[j] / (p - 1) * w[j] + ((p - u[j]) / (p - 1) * w[j - 1] if j else 0) for j in range(ORDER)]
        return lo.long(), torch.stack(w, -1)

    def nodes(self, x):
        lo, w = self.bspline(x)
        N = self.prm["Nb"]
        k = torch.arange(ORDER, device=self.dev)
        i = [(lo[:, d, None] + k) % N[d] for d in range(3)]
        node = i[0][:, None, None] + N[0] * (i[1][:, None, :, None] + N[1] * i[2][:, :, None, None])
        return node.flatten(1), (w[:, 2, :, None, None] * w[:, 1, None, :, None] * w[:, 0, None, None]).flatten(1)

    def mesh(self, v, x):
        N1, N2, N3 = self.prm["Nb"]
        X = self.pts(self.X).reshape(-1, 3)
        src = [self.c1 * self.pts(self.dF).reshape(-1, 3)]
        if self.c2:
            g, n = self.pts(self.dG).reshape(-1, 3), self.pts(self.N).reshape(-1, 3)
            src += [self.c2 * g * n[:, j, None] for j in range(3)]
        src = torch.cat(src, 1)
        H = torch.zeros(src.shape[1], N1 * N2 * N3, dtype=torch.float64, device=self.dev)
        for q in torch.arange(X.shape[0], device=self.dev).split(40000):
            node, w = self.nodes(X[q])
            for k in range(src.shape[1]):
                H[k].index_add_(0, node.flatten(), (w * src[q, k, None]).flatten())
        H = torch.stack([torch.fft.rfftn(h.reshape(N3, N2, N1)) for h in H])  # (.., kz, ky, kx)
        f = [torch.arange(n, dtype=torch.float64, device=self.dev) for n in (N1 // 2 + 1, N2, N3)]
        qx = (f[0] / self.L[0])[None, None]
        qy = (torch.where(f[1] < N2 // 2, f[1], f[1] - N2) / self.L[1])[None, :, None]
        qz = (torch.where(2 * f[2] <= N3, f[2], f[2] - N3) / self.L[2])[:, None, None]
        q = torch.stack(torch.broadcast_tensors(qx, qy, qz))
        a, vol = self.prm["alpha"], float(self.L.prod())
        q2 = math.pi * a * (q * q).sum(0)
        q2[0, 0, 0] = 1.0
        e = (-q2).exp()
        p0 = e / q2
        p1 = (e + p0) / q2
        qt = math.sqrt(math.pi * a) * q
        V = 2 * a / vol * p1 * (q2 * H[:3] - qt * (qt * H[:3]).sum(0))
        if self.c2:
            T = H[3:].reshape(3, 3, *H.shape[1:]).transpose(0, 1)  # T[g component][normal component]
            s0, s1 = 4 * math.pi * a / vol * p0, 8 * math.pi ** 2 * a * a / vol * p1
            wv = q * (T[0, 0] + T[1, 1] + T[2, 2]) + torch.einsum("azyx,abzyx->bzyx", q.to(T.dtype), T) + torch.einsum("azyx,bazyx->bzyx", q.to(T.dtype), T)
            V = V - 1j * (s0 * wv - s1 * torch.einsum("azyx,abzyx,bzyx->zyx", q.to(T.dtype), T, q.to(T.dtype)) * q)
        u = torch.arange(ORDER - 1, dtype=torch.float64, device=self.dev)
        M = self.bspline(torch.zeros(1, 3, dtype=torch.float64, device=self.dev))[1][0, 0]
        M = M[: ORDER - 1]
        bb = []
        for n, k in ((N1, f[0]), (N2, f[1]), (N3, f[2])):
            z = (M * torch.exp(2j * math.pi * k[:, None] * u / n)).sum(1)
            bb.append(1 / z.abs() ** 2)
        V = V * (bb[0][None, None] * bb[1][None, :, None] * bb[2][:, None, None])
        V[:, 0, 0, 0] = 0
        for i in (0, N1 // 2) if N1 % 2 == 0 else (0,):  # a real field's planes
            p = V[..., i]
            mirror = torch.roll(p.flip(1, 2), (1, 1), (1, 2)).conj()
            V[..., i] = 0.5 * (p + mirror)
        U = torch.fft.irfftn(V, s=(N3, N2, N1), dim=(1, 2, 3), norm="forward").reshape(3, -1)
        for q in torch.arange(x.shape[0], device=self.dev).split(100000):
            node, w = self.nodes(x[q])
            v[q] += torch.stack([(U[k][node] * w).sum(1) for k in range(3)], 1)


def exact(case, seed):
    """The sums of a matvec, a step or a field.  None for the solves, whose
    outputs are whatever meets the tolerance first, and for suspensions that
    would take too long."""
    if case["kind"] in ("cell", "wall") or case["ncell"] * case["nlat"] * case["nlon"] > 400000:
        return None
    E = _Exact(case, seed)
    if case["kind"] == "field":
        x = E.t(E.s.points).T.contiguous()
        A = torch.full_like(x[:, 0], 2.0)
    else:
        x, A = E.pts(E.X).reshape(-1, 3), E.A.repeat_interleave(E.nv)
    v = E.velocity(x, A, own=case["kind"] != "field")
    if case["kind"] == "field":
        v = v + E.t(E.prm["vBkg"])
    return v.T.cpu().numpy()
