"""What the framework's performance is measured on: the calls of a CheFSI SCF through the
library's public entry points, over the range of sizes its configurations, tests and benchmark
name. Each case is one call (or the few calls of one step) as a program makes them.

Kinds of case:
  filter     ChebyshevFiltering on real orbital blocks: FP64 and FP32 device blocks, and host
             arrays as SPARC passes them (X input only, the form eigSolve_CheFSI needs)
  apply      Hamiltonian_vectors_mult (the Lanczos bounds, the residual checks and H Y call it)
  subspace   the Rayleigh-Ritz products around the filter: Project_Hamiltonian, then
             Subspace_Rotation
  kfilter    ChebyshevFiltering_batched over (k-point, spin) blocks of complex orbitals
  poisson    Calculate_elecstPotential (the AAR solve of every SCF iteration)
  scf        a whole single-point SCF from the atomic densities of a diamond Si cell
"""
import math
import os

import numpy as np
import torch

import sparc_gb300 as sg
from sparc_gb300.psp8 import load_tables
from sparc_gb300.setup import CellSystem
from sparc_gb300.synthetic import fd_d2_coeffs, gaussian_potential, real_ylm

SI_A = 10.26     # Bohr, conventional cubic cell of diamond Si
DIAMOND = np.array([[0.00, 0.00, 0.00], [0.00, 0.50, 0.50], [0.50, 0.00, 0.50],
                    [0.50, 0.50, 0.00], [0.25, 0.25, 0.25], [0.25, 0.75, 0.75],
                    [0.75, 0.25, 0.75], [0.75, 0.75, 0.25]])
# filter bounds: those of the stencil/filter microbenchmark
CUT, HIGH, LOW = 0.5, 50.0, -1.0


def _filter(name, n, h, ncol, degree, natom, rc, nproj, dtype="f64", where="device"):
    return dict(name=name, kind="filter", nx=n[0], ny=n[1], nz=n[2], h=h, ncol=ncol,
                degree=degree, natom=natom, rc=rc, nproj=nproj, dtype=dtype, where=where)


def listed():
    return [
        # a 2-atom cell, the smallest calls a user makes: a few columns on a 14^3 grid
        _filter("filter 14^3 x 8 f64", (14, 14, 14), 0.5, 8, 16, 2, 1.93, 18),
        # the 8-atom Si cell of the plain FP64 SCF: 26^3, 32 states
        _filter("filter 26^3 x 32 f64", (26, 26, 26), 0.3946, 32, 20, 8, 1.93, 18),
        # the stencil/filter microbenchmark in the reference's precision
        _filter("filter 96^3 x 512 f64", (96, 96, 96), 0.35, 512, 20, 64, 6.0, 9),
        # the same block in the mixed mode's precision, resident in FP32
        _filter("filter 96^3 x 512 f32", (96, 96, 96), 0.35, 512, 20, 64, 6.0, 9, dtype="f32"),
        # SPARC's own arrays (pageable host memory) through the drop-in call: 64-atom Si cell
        _filter("filter 52^3 x 160 f64 host", (52, 52, 52), 0.3946, 160, 20, 64, 1.93, 18,
                where="host"),
        # H applied to an odd number of columns on a ragged cell
        dict(name="apply 61x45x53 x 37 f64", kind="apply", nx=61, ny=45, nz=53, h=0.4, ncol=37,
             natom=60, rc=1.93, nproj=18),
        # the Rayleigh-Ritz products of the 216-atom Si cell, FP64 and the mixed mode's FP32
        dict(name="subspace 77^3 x 520 f64", kind="subspace", nx=77, ny=77, nz=77, h=0.4,
             ncol=520, natom=216, rc=1.93, nproj=18, dtype="f64"),
        dict(name="subspace 77^3 x 520 f32", kind="subspace", nx=77, ny=77, nz=77, h=0.4,
             ncol=520, natom=216, rc=1.93, nproj=18, dtype="f32"),
        # 32-atom Al, 10 k-points x 2 spins of 64 states, in both precisions of the filter
        dict(name="kfilter 34^3 x 20x64 c128", kind="kfilter", nx=34, ny=34, nz=34, h=0.45,
             ncol=64, nk=10, nspin=2, degree=18, natom=32, rc=1.96, nproj=18, dtype="c128"),
        dict(name="kfilter 34^3 x 20x64 c64", kind="kfilter", nx=34, ny=34, nz=34, h=0.45,
             ncol=64, nk=10, nspin=2, degree=18, natom=32, rc=1.96, nproj=18, dtype="c64"),
        # the electrostatic potential of the 216-atom cell
        dict(name="poisson 77^3", kind="poisson", nx=77, ny=77, nz=77, h=0.4, natom=216,
             tol=1e-8),
        # a whole SCF of the 8-atom Si cell (26^3, 32 states) to 1e-6
        dict(name="scf Si8 f64", kind="scf", states=32, degree=20, sigma=0.05, mesh=0.40),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _grid(rng, lo, hi):
    """Near-cubic grid with ragged edges."""
    n = _log(rng, lo, hi)
    return [max(12, min(hi, int(round(n * rng.uniform(0.85, 1.15))))) for _ in range(3)]


def draw(rng):
    kind = rng.choice(["filter", "filter", "filter", "apply", "subspace", "kfilter", "poisson",
                       "scf"])
    if kind == "scf":
        return dict(kind="scf", states=rng.randint(22, 34), degree=rng.randint(16, 22),
                    sigma=round(rng.uniform(0.02, 0.1), 3), mesh=round(rng.uniform(0.42, 0.55), 3))
    h = round(rng.uniform(0.33, 0.5), 4)
    if kind == "poisson":
        nx, ny, nz = _grid(rng, 20, 90)
        return dict(kind="poisson", nx=nx, ny=ny, nz=nz, h=h,
                    natom=max(2, nx * ny * nz // 2100), tol=1e-8)
    if kind == "kfilter":
        nx, ny, nz = _grid(rng, 14, 40)
        c = dict(kind="kfilter", nx=nx, ny=ny, nz=nz, h=h, ncol=int(_log(rng, 6, 72)),
                 nk=rng.randint(1, 10), nspin=rng.randint(1, 2), degree=rng.randint(12, 20),
                 natom=max(2, nx * ny * nz // 1200), rc=1.96, nproj=18,
                 dtype=rng.choice(["c128", "c64"]))
        return c
    nx, ny, nz = _grid(rng, 14, 90)
    nd = nx * ny * nz
    ncol = int(_log(rng, 4, 520))
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, h=h, ncol=ncol, natom=max(2, nd // 2100), rc=1.93,
             nproj=18)
    if kind == "filter":
        c["degree"] = rng.randint(12, 24)
        c["dtype"] = rng.choice(["f64", "f64", "f32"])
        c["where"] = rng.choice(["device", "device", "host"])
        if c["where"] == "host":
            c["dtype"] = "f64"
        if rng.random() < 0.3:  # larger spheres, as the microbenchmark's
            c.update(rc=round(rng.uniform(3.0, 6.0), 2), nproj=9, natom=max(1, nd // 14000))
        most = (1 << 27) if c["where"] == "device" else (1 << 25)
        c["ncol"] = max(4, min(ncol, most // nd))
    elif kind == "subspace":
        c["dtype"] = rng.choice(["f64", "f32"])
        c["ncol"] = max(8, ncol)
    return c


# ------------------------------------------------------------------ inputs

def _projectors(rng, N, h, natom, rc, nproj):
    """Atoms on random sites, nproj Kleinman-Bylander projectors each (l = 0, 1, 2; one radial
    function per l for 9, two for 18), split into the atom's periodic images as a SPARC set-up
    splits them: image g of an atom holds the points of its sphere that lie in one copy of the
    cell. Returns the set_nonlocal arrays and the image coordinates of set_kpoint_geometry."""
    N = np.asarray(N)
    L = N * h
    nr = int(math.ceil(rc / h)) + 1
    off = np.arange(-nr, nr + 1)
    OZ, OY, OX = (o.reshape(-1) for o in np.meshgrid(off, off, off, indexing="ij"))
    off3 = np.stack([OX, OY, OZ], axis=1)
    pos = rng.uniform(0.0, 1.0, size=(natom, 3)) * L
    per_l = nproj // 9
    gam = rng.uniform(-2.0, 4.0, size=(3, per_l))
    gamma = np.concatenate([np.repeat(gam[l, p], 2 * l + 1) for l in range(3)
                            for p in range(per_l)])
    img_atom, img_ndc, grid_pos, chi, coords = [], [], [], [], []
    for a in range(natom):
        g = np.floor(pos[a] / h).astype(int) + off3
        d = g * h - pos[a]
        r = np.sqrt((d * d).sum(axis=1))
        keep = r <= rc
        g, d, r = g[keep], d[keep], r[keep]
        cols = []
        for l in range(3):
            ylm = real_ylm(l, d[:, 0], d[:, 1], d[:, 2], r)
            for _ in range(per_l):
                c = rng.uniform(0.5, 1.5, size=3)
                u = (c[0] + c[1] * (r / rc) + c[2] * (r / rc) ** 2) * \
                    np.cos(0.5 * math.pi * r / rc) ** 2 * (r / rc) ** l
                cols += [u * y for y in ylm]
        table = np.stack(cols, axis=0)
        cell = np.floor_divide(g, N)          # which copy of the cell a point lies in
        w = g - cell * N
        p = w[:, 0] + N[0] * (w[:, 1] + N[1] * w[:, 2])
        for shift in np.unique(cell, axis=0):
            m = np.flatnonzero((cell == shift).all(axis=1))
            m = m[np.argsort(p[m], kind="stable")]
            img_atom.append(a)
            img_ndc.append(len(m))
            grid_pos.append(p[m])
            chi.append(table[:, m].reshape(-1))
            coords.append(pos[a] - shift * L)  # the image whose sphere reaches into the cell
    return dict(ip_displ=np.arange(natom + 1, dtype=np.int32) * nproj,
                gamma=np.tile(gamma, natom), img_atom=np.array(img_atom, dtype=np.int32),
                img_ndc=np.array(img_ndc, dtype=np.int32),
                grid_pos=np.concatenate(grid_pos).astype(np.int32),
                chi=np.concatenate(chi)), np.array(coords)


def _system(case, seed):
    """Local potential and projectors of a case: plain arrays, made from the seed."""
    N, h = (case["nx"], case["ny"], case["nz"]), case["h"]
    rng = np.random.default_rng(seed)
    veff = gaussian_potential(rng, N, h, ncenters=min(64, max(4, case["natom"])))
    nl, coords = _projectors(rng, N, h, case["natom"], case["rc"], case["nproj"])
    return N, h, veff, nl, coords


def _context(N, h, veff, nl, nspin=1):
    c = fd_d2_coeffs(6, h)
    ctx = sg.Context(*N, 6, c, c, c, h ** 3)
    ctx.set_veff(veff, nspin=nspin)
    if nl is not None:
        ctx.set_nonlocal(nl["ip_displ"], nl["gamma"], nl["img_atom"], nl["img_ndc"],
                         nl["grid_pos"], nl["chi"])
    return ctx


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _rand(shape, gen, dtype):
    return torch.rand(shape, generator=gen, device="cuda", dtype=dtype).mul_(2).sub_(1)


def _subspace_blocks(case, seed):
    """A filtered block and the matrix that rotates it: the filter amplifies each state by its
    own factor, and the eigenvectors undo that."""
    gen = _gen(seed)
    dt = torch.float32 if case["dtype"] == "f32" else torch.float64
    ns, nd = case["ncol"], case["nx"] * case["ny"] * case["nz"]
    scale = 10.0 ** (2.0 * _rand((ns,), gen, torch.float64))
    Y = _rand((ns, nd), gen, dt)
    Y *= scale.to(dt)[:, None]
    Q = _rand((ns, ns), gen, torch.float64) / (math.sqrt(ns) * scale[None, :])
    return Y, Q


def _kblocks(case, seed):
    """(spin, k, X) of every block: k-points of a 4 x 4 x 4 grid, spins alternating."""
    gen = _gen(seed)
    rng = np.random.default_rng(seed + 1)
    nd = case["nx"] * case["ny"] * case["nz"]
    L = np.array([case["nx"], case["ny"], case["nz"]]) * case["h"]
    real = torch.float32 if case["dtype"] == "c64" else torch.float64
    out = []
    for _ in range(case["nk"]):
        k = 2 * np.pi / L * rng.integers(0, 3, size=3) / 4
        for spin in range(case["nspin"]):
            x = _rand((case["ncol"], nd, 2), gen, real)
            out.append((spin, [float(v) for v in k], torch.view_as_complex(x)))
    return out


def _charges(case, seed):
    """A smooth electron density and the neutralising pseudocharge of the same centres, narrower
    (the right side of the electrostatic problem of a cell)."""
    N, h = (case["nx"], case["ny"], case["nz"]), case["h"]
    n = min(64, case["natom"])
    rho = -gaussian_potential(np.random.default_rng(seed), N, h, ncenters=n, amp=-1.0, width=1.8)
    b = gaussian_potential(np.random.default_rng(seed), N, h, ncenters=n, amp=-1.0, width=1.0)
    b *= -rho.sum() / b.sum()
    return rho, b


def prepare(case, seed):
    kind = case["kind"]
    if kind == "scf":
        rng = np.random.default_rng(seed)
        tables = load_tables(os.path.join("tests", "golden", "psp_Si.npz"))
        pos = DIAMOND * SI_A + rng.normal(0.0, case["sigma"], size=(8, 3))
        n = int(math.ceil(SI_A / case["mesh"]))
        cs = CellSystem((SI_A,) * 3, (n,) * 3, [("Si", pos)], {"Si": tables})
        return dict(kind=kind, cs=cs, params=cs.scf_params(case["states"], case["degree"]))
    if kind == "poisson":
        rho, b = _charges(case, seed)
        ctx = _context((case["nx"], case["ny"], case["nz"]), case["h"], rho * 0, None)
        return dict(kind=kind, ctx=ctx, tol=case["tol"], rho=torch.from_numpy(rho).cuda(),
                    b=torch.from_numpy(b).cuda())
    N, h, veff, nl, coords = _system(case, seed)
    nd = N[0] * N[1] * N[2]
    if kind == "kfilter":
        spins = [veff + 0.02, veff - 0.02][:case["nspin"]]
        ctx = _context(N, h, np.concatenate(spins), nl, nspin=case["nspin"])
        ctx.set_kpoint_geometry([n * h for n in N], coords)
        blocks = [dict(spin=s, k=k, X=x.clone(), Y=torch.empty_like(x), X0=x, a=CUT, b=HIGH,
                       a0=LOW) for s, k, x in _kblocks(case, seed)]
        return dict(kind=kind, ctx=ctx, blocks=blocks, degree=case["degree"],
                    precision=sg.SGPU_PREC_FP32 if case["dtype"] == "c64" else sg.SGPU_PREC_FP64)
    ctx = _context(N, h, veff, nl)
    if kind == "subspace":
        Y, Q = _subspace_blocks(case, seed)
        ns = case["ncol"]
        if case["dtype"] == "f32":
            ctx.autotune(ncol=ns)
        return dict(kind=kind, ctx=ctx, dtype=case["dtype"], Y=Y, Q=Q, HY=torch.empty_like(Y),
                    X=torch.empty_like(Y), Hp=torch.empty_like(Q), Mp=torch.empty_like(Q))
    st = dict(kind=kind, ctx=ctx, degree=case.get("degree"), dtype=case.get("dtype", "f64"))
    if case.get("where") == "host":
        st["kind"] = "hostfilter"
        st["X"] = _host_block(case, seed)
        st["Y"] = np.zeros_like(st["X"])
        return st
    if case.get("dtype") == "f32":
        ctx.autotune(ncol=case["ncol"])  # as the mixed-mode SCF does before its first filter
    st["X0"] = _rand((case["ncol"], nd), _gen(seed),
                     torch.float32 if st["dtype"] == "f32" else torch.float64)
    st["X"], st["Y"] = st["X0"].clone(), torch.empty_like(st["X0"])
    return st


def _host_block(case, seed):
    nd = case["nx"] * case["ny"] * case["nz"]
    return np.random.default_rng(seed).uniform(-1.0, 1.0, size=(case["ncol"], nd))


def run(s):
    kind = s["kind"]
    if kind == "scf":
        res, rho, lam, occ = s["cs"].scf(s["params"])
        return res["Etot"], rho, lam, occ
    ctx = s["ctx"]
    if kind == "filter":
        s["X"].copy_(s["X0"])  # the filter works in place on the block that the rotation wrote
        f = ctx.ChebyshevFiltering_f32 if s["dtype"] == "f32" else ctx.ChebyshevFiltering
        f(s["X"], s["Y"], s["degree"], CUT, HIGH, LOW)
        return s["X"], s["Y"]
    if kind == "hostfilter":
        ctx.ChebyshevFiltering_y(s["X"], s["Y"], s["degree"], CUT, HIGH, LOW)
        return s["Y"]
    if kind == "apply":
        ctx.Hamiltonian_vectors_mult(-0.3, s["X0"], s["Y"])
        return s["Y"]
    if kind == "subspace":
        if s["dtype"] == "f32":
            ctx.Project_Hamiltonian_f32(s["Y"], s["HY"], s["Hp"], s["Mp"])
            ctx.Subspace_Rotation_f32(s["Y"], s["Q"], s["X"])
        else:
            ctx.Project_Hamiltonian(s["Y"], s["HY"], s["Hp"], s["Mp"])
            ctx.Subspace_Rotation(s["Y"], s["Q"], s["X"])
        return s["HY"], s["Hp"], s["Mp"], s["X"]
    if kind == "kfilter":
        for b in s["blocks"]:
            b["X"].copy_(b["X0"])
        ctx.ChebyshevFiltering_batched(s["blocks"], s["degree"], precision=s["precision"])
        return [(b["X"], b["Y"]) for b in s["blocks"]]
    phi = torch.zeros_like(s["rho"])
    ctx.Calculate_elecstPotential(s["rho"], s["b"], phi, s["tol"])
    return phi


# ------------------------------------------------------------------ work

def work(case):
    kind = case["kind"]
    if kind == "scf":  # about 14 iterations, 4 filter passes in the first
        n = int(math.ceil(SI_A / case["mesh"])) ** 3
        return dict(bytes=n * 8 * 20, flops=17.0 * case["degree"] * n * case["states"] * 120)
    nd = case["nx"] * case["ny"] * case["nz"]
    if kind == "poisson":
        return dict(bytes=nd * 8 * 3, flops=nd * 61.0 * 60)
    ncol = case["ncol"]
    pairs = case["natom"] * case["nproj"] * 4.0 / 3.0 * math.pi * (case["rc"] / case["h"]) ** 3
    apply = 61.0 * nd + 4.0 * pairs   # one H x: stencil, recurrence, projection and its apply
    if kind == "filter":
        size = 4 if case["dtype"] == "f32" else 8
        return dict(bytes=(3.0 if case["where"] == "device" else 2.0) * nd * ncol * size + 8 * nd
                    + 8 * pairs, flops=case["degree"] * ncol * apply)
    if kind == "apply":
        return dict(bytes=2.0 * nd * ncol * 8 + 8 * nd + 8 * pairs, flops=ncol * apply)
    if kind == "subspace":
        size = 4 if case["dtype"] == "f32" else 8
        return dict(bytes=3.0 * nd * ncol * size + 3 * 8 * ncol * ncol,
                    flops=ncol * apply + 5.0 * nd * ncol * ncol)
    cols = ncol * case["nk"] * case["nspin"]
    size = 8 if case["dtype"] == "c64" else 16
    return dict(bytes=3.0 * nd * cols * size, flops=case["degree"] * 2.0 * cols * apply)


# ------------------------------------------------------------------ 64-bit values

class _Exact:
    """H x in 64 bits with plain torch; columns in rows, grid x fastest."""

    def __init__(self, N, h, veff, nl, coords=None, k=None):
        self.N, self.c, self.dV = N, fd_weights(h), h ** 3
        self.veff = torch.from_numpy(veff).cuda()
        self.k, self.L = k, np.array(N) * h
        self.gamma = torch.from_numpy(nl["gamma"]).cuda()
        self.images, g0, c0 = [], 0, 0
        for i, (a, n) in enumerate(zip(nl["img_atom"], nl["img_ndc"])):
            r0, r1 = int(nl["ip_displ"][a]), int(nl["ip_displ"][a + 1])
            chi = nl["chi"][c0:c0 + n * (r1 - r0)].reshape(r1 - r0, n)
            theta = 0.0 if k is None else -float(np.dot(k, np.floor(coords[i] / self.L) * self.L))
            self.images.append((r0, r1, torch.from_numpy(nl["grid_pos"][g0:g0 + n].astype(
                np.int64)).cuda(), torch.from_numpy(np.ascontiguousarray(chi)).cuda(), theta))
            g0, c0 = g0 + n, c0 + n * (r1 - r0)

    def _shifted(self, v, axis, r):
        """v at the points r further along an axis (1 z, 2 y, 3 x), with the Bloch factor of the
        cell that they lie in."""
        out = torch.roll(v, -r, dims=axis)
        if self.k is None:
            return out
        d = 3 - axis
        n, kl = self.N[d], float(self.k[d] * self.L[d])
        i = torch.arange(n, device=v.device) + r
        ph = torch.polar(torch.ones(n, device=v.device, dtype=torch.float64),
                         kl * torch.div(i, n, rounding_mode="floor").double())
        return out * ph.reshape([n if a == axis else 1 for a in range(4)])

    def apply(self, x, c):
        nx, ny, nz = self.N
        v = x.reshape(-1, nz, ny, nx)
        y = (-1.5 * self.c[0] + c + self.veff).reshape(1, nz, ny, nx) * v
        for axis in (1, 2, 3):
            for r in range(1, 7):
                t = self._shifted(v, axis, r)
                t += self._shifted(v, axis, -r)
                y.add_(t, alpha=-0.5 * float(self.c[r]))
        y = y.reshape(x.shape)
        alpha = torch.zeros((x.shape[0], self.gamma.numel()), device=x.device, dtype=x.dtype)
        for r0, r1, pos, chi, theta in self.images:
            ph = complex(math.cos(theta), math.sin(theta)) if self.k is not None else 1.0
            alpha[:, r0:r1] += (ph * self.dV) * (x[:, pos] @ chi.T.to(x.dtype))
        alpha *= self.gamma
        for r0, r1, pos, chi, theta in self.images:
            ph = complex(math.cos(theta), -math.sin(theta)) if self.k is not None else 1.0
            y.index_add_(1, pos, ph * (alpha[:, r0:r1] @ chi.to(x.dtype)))
        return y

    def filter(self, x, m):
        """The degree m-1 and degree m iterates of the scaled Chebyshev filter."""
        e, c = 0.5 * (HIGH - CUT), 0.5 * (HIGH + CUT)
        sigma = e / (LOW - c)
        gamma = 2.0 / sigma
        prev, cur = x, self.apply(x, -c) * (sigma / e)
        for _ in range(1, m):
            s2 = 1.0 / (gamma - sigma)
            nxt = self.apply(cur, -c) * (2.0 * s2 / e)
            nxt.sub_(prev, alpha=sigma * s2)
            prev, cur, sigma = cur, nxt, s2
        return prev, cur


def fd_weights(h):
    """Second-derivative weights of order 12 divided by h^2."""
    f = math.factorial
    w = [sum(-2.0 / (p * p) for p in range(1, 7))]
    w += [2.0 * (-1) ** (p + 1) * f(6) * f(6) / (f(6 - p) * f(6 + p)) / (p * p)
          for p in range(1, 7)]
    return np.array(w) / (h * h)


def _by_columns(x, nd, f):
    """f over groups of columns, so that the 64-bit intermediates stay small."""
    step = max(1, int(2e8 // nd))
    parts = [f(x[i:i + step]) for i in range(0, x.shape[0], step)]
    if isinstance(parts[0], tuple):
        return tuple(torch.cat(p) for p in zip(*parts))
    return torch.cat(parts)


def exact(case, seed):
    kind = case["kind"]
    if kind == "scf":
        return None
    if kind == "poisson":
        rho, b = _charges(case, seed)
        N, c = (case["nz"], case["ny"], case["nx"]), fd_weights(case["h"])
        lap = torch.zeros(N, dtype=torch.float64, device="cuda")
        for axis, n in enumerate(N):
            t = 2 * np.pi * np.arange(n) / n
            lam = c[0] + sum(2 * c[r] * np.cos(r * t) for r in range(1, 7))
            lap += torch.from_numpy(lam).cuda().reshape([n if a == axis else 1 for a in range(3)])
        f = torch.fft.fftn(torch.from_numpy(4 * np.pi * (rho + b)).cuda().reshape(N))
        lap[0, 0, 0] = 1.0
        f = f / -lap
        f[0, 0, 0] = 0.0
        return torch.fft.ifftn(f).real.reshape(-1).contiguous()
    N, h, veff, nl, coords = _system(case, seed)
    nd = N[0] * N[1] * N[2]
    if kind == "kfilter":
        out = []
        for spin, k, x in _kblocks(case, seed):
            ex = _Exact(N, h, veff + (0.02 if spin == 0 else -0.02), nl, coords, k)
            out.append(ex.filter(x.to(torch.complex128), case["degree"]))
        return out
    ex = _Exact(N, h, veff, nl)
    if kind == "subspace":
        Y, Q = _subspace_blocks(case, seed)
        Y = Y.double()
        HY = _by_columns(Y, nd, lambda x: ex.apply(x, 0.0))
        return HY, HY @ Y.T, Y @ Y.T, Q @ Y
    if case.get("where") == "host":
        X = torch.from_numpy(_host_block(case, seed)).cuda()
        return _by_columns(X, nd, lambda x: ex.filter(x, case["degree"])[1])
    X = _rand((case["ncol"], nd), _gen(seed),
              torch.float32 if case.get("dtype") == "f32" else torch.float64).double()
    if kind == "apply":
        return _by_columns(X, nd, lambda x: ex.apply(x, -0.3))
    return _by_columns(X, nd, lambda x: ex.filter(x, case["degree"]))
