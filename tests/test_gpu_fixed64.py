"""FP64 kernels in block fixed point (csrc/fixed64.cuh) at the sizes and values where they can go
wrong: tiles cut by the grid edge, rows that wrap several times, slabs, fields whose largest value
grows along z (a new block scale), columns that the fixed-point range does not cover."""
import numpy as np
import pytest

import sparc_gb300 as sg
from oracle.oracle import Oracle
from sparc_gb300.synthetic import fd_d2_coeffs, synthetic_nonlocal

pytestmark = pytest.mark.gpu


def _fields(N, rng):
    Nd = N[0] * N[1] * N[2]
    z = np.arange(Nd) // (N[0] * N[1])
    u = rng.uniform(-1, 1, (2, Nd))
    return {"uniform": u, "growing": u * 2.0 ** (1.5 * z), "falling": u * 2.0 ** (-1.5 * z),
            "one point": np.eye(1, Nd, Nd // 2) * 3.7, "zero": np.zeros((1, Nd)),
            "wide": u * 10.0 ** rng.uniform(-12, 0, (2, Nd)), "tiny": u * 1e-290,
            "huge": u * 1e290}


@pytest.mark.parametrize("N", [(14, 14, 14), (6, 7, 9), (31, 17, 23), (45, 33, 12), (34, 12, 70),
                               (77, 20, 13)])
@pytest.mark.parametrize("h", [(0.4, 0.4, 0.4), (0.4, 0.37, 0.45)])
def test_stencil_fields(gpu_available, N, h):
    """Both weight forms (equal and different spacings). Each result is off by at most the
    rounding of the oracle's 37-term sum and the two final operations, 40 units of 2^-53 of the
    sum of |coefficient| times the column's largest value."""
    rng = np.random.default_rng(sum(N))
    c = [fd_d2_coeffs(6, x) for x in h]
    grid = dict(Nx=N[0], Ny=N[1], Nz=N[2], FDn=6, cx=c[0], cy=c[1], cz=c[2], dV=float(np.prod(h)))
    ctx = sg.Context(*N, 6, *c, grid["dV"])
    o = Oracle(grid, None)
    Nd = N[0] * N[1] * N[2]
    v = rng.normal(size=Nd)
    S = 0.5 * sum(abs(w[0]) + 2 * np.abs(w[1:]).sum() for w in c) + 3.1 + np.abs(v).max()
    for name, x in _fields(N, rng).items():
        y = np.full_like(x, np.nan)
        ctx.Lap_plus_diag_vec_mult_orth(-0.5, 1.0, -3.1, v, x, y)
        ref = o.lap_plus_diag(-0.5, 1.0, -3.1, v, x)
        for n in range(x.shape[0]):
            assert np.abs(y[n] - ref[n]).max() <= 40 * 2.0 ** -53 * S * np.abs(x[n]).max(), name
    ctx.close()


@pytest.mark.parametrize("N", [(14, 14, 14), (6, 7, 9), (31, 17, 23), (45, 33, 12), (34, 12, 70),
                               (77, 20, 13)])
@pytest.mark.parametrize("h", [(0.4, 0.4, 0.4), (0.4, 0.37, 0.45)])
def test_stencil_fields_many_columns(gpu_available, N, h):
    """The same fields and bound in calls of at least 120000 points and columns, above the sizes
    that the point-per-thread kernel takes: the fields' columns in turn."""
    rng = np.random.default_rng(sum(N))
    c = [fd_d2_coeffs(6, x) for x in h]
    grid = dict(Nx=N[0], Ny=N[1], Nz=N[2], FDn=6, cx=c[0], cy=c[1], cz=c[2], dV=float(np.prod(h)))
    ctx = sg.Context(*N, 6, *c, grid["dV"])
    o = Oracle(grid, None)
    Nd = N[0] * N[1] * N[2]
    v = rng.normal(size=Nd)
    S = 0.5 * sum(abs(w[0]) + 2 * np.abs(w[1:]).sum() for w in c) + 3.1 + np.abs(v).max()
    cols = np.concatenate(list(_fields(N, rng).values()))
    x = np.ascontiguousarray(np.resize(cols, (max(len(cols), -(-120000 // Nd)), Nd)))
    y = np.full_like(x, np.nan)
    ctx.Lap_plus_diag_vec_mult_orth(-0.5, 1.0, -3.1, v, x, y)
    ref = o.lap_plus_diag(-0.5, 1.0, -3.1, v, cols)
    for n in range(x.shape[0]):
        tol = 40 * 2.0 ** -53 * S * np.abs(x[n]).max()
        assert np.abs(y[n] - ref[n % len(cols)]).max() <= tol
    ctx.close()


@pytest.mark.parametrize("scale", [1.0, 1e3, 1e9, 0.0])
def test_stencil_potential_range(gpu_available, scale):
    """A potential of the stencil's own size, one far above it (the FP64 kernel takes over) and
    none; the filter's recurrence term; a few columns and enough columns for whole-z slabs."""
    N, h = (20, 18, 26), 0.4
    rng = np.random.default_rng(5)
    c = fd_d2_coeffs(6, h)
    grid = dict(Nx=N[0], Ny=N[1], Nz=N[2], FDn=6, cx=c, cy=c, cz=c, dV=h ** 3)
    ctx = sg.Context(*N, 6, c, c, c, h ** 3)
    o = Oracle(grid, None)
    Nd = N[0] * N[1] * N[2]
    v = rng.normal(size=Nd) * scale
    ctx.set_veff(v)
    S = 1.5 * (abs(c[0]) + 2 * np.abs(c[1:]).sum()) + 20 + np.abs(v).max()
    for ncol in (1, 3, 300):
        x = rng.uniform(-1, 1, (ncol, Nd))
        y = np.zeros_like(x)
        ctx.Hamiltonian_vectors_mult(-20.0, x, y)
        k = min(ncol, 3)
        assert np.abs(y[:k] - o.hamiltonian(v, -20.0, x[:k])).max() <= 40 * 2.0 ** -53 * S
        b = 2.0 * S  # above the spectrum: the recurrence keeps the block near its input's size
        X, Y = x.copy(), np.zeros_like(x)
        ctx.ChebyshevFiltering(X, Y, 4, 0.1 * S, b, -b)
        Xo, Yo = o.chebyshev(v, 4, 0.1 * S, b, -b, x[:k])
        # four applies, each scaled to at most 4, on iterates at most 8 times the input
        assert np.abs(Y[:k] - Yo).max() <= 4 * 4 * 8 * 40 * 2.0 ** -53
        assert np.abs(X[:k] - Xo).max() <= 4 * 4 * 8 * 40 * 2.0 ** -53
    ctx.close()


@pytest.mark.parametrize("reps", [1, 4])
def test_stencil_nonfinite(gpu_available, reps):
    """An infinity and a NaN reach exactly the points whose stencil touches them; below and above
    the sizes of the point-per-thread kernel."""
    N, h = (33, 21, 30), 0.4
    rng = np.random.default_rng(6)
    c = fd_d2_coeffs(6, h)
    grid = dict(Nx=N[0], Ny=N[1], Nz=N[2], FDn=6, cx=c, cy=c, cz=c, dV=h ** 3)
    ctx = sg.Context(*N, 6, c, c, c, h ** 3)
    Nd = N[0] * N[1] * N[2]
    x = rng.uniform(-1, 1, (3, Nd))
    x[0, Nd // 3] = np.nan
    x[1, Nd // 2] = np.inf
    x[2, 7] = -np.inf
    x = np.tile(x, (reps, 1))
    y = np.zeros_like(x)
    ctx.Lap_vec_mult(0.3, x, y)
    ref = np.tile(Oracle(grid, None).lap_plus_diag(1.0, 0.0, 0.3, None, x[:3]), (reps, 1))
    fin = np.isfinite(ref)
    assert np.array_equal(np.isfinite(y), fin) and np.array_equal(np.isnan(y), np.isnan(ref))
    S = 3 * (abs(c[0]) + 2 * np.abs(c[1:]).sum()) + 0.3
    assert np.abs((y - ref)[fin]).max() <= 40 * 2.0 ** -53 * S
    ctx.close()


def _nonlocal_case(N, h, natom, rc, lmax, seed, dup=1):
    """Grid, potential and projectors; dup > 1 doubles the projectors of every atom."""
    rng = np.random.default_rng(seed)
    c = fd_d2_coeffs(6, h)
    grid = dict(Nx=N[0], Ny=N[1], Nz=N[2], FDn=6, cx=c, cy=c, cz=c, dV=h ** 3)
    nl = synthetic_nonlocal(rng, N, h, natom=natom, rc=rc, lmax=lmax)
    if dup > 1:
        np1 = (lmax + 1) ** 2
        nl["ip_displ"] = nl["ip_displ"] * dup
        nl["gamma"] = np.tile(nl["gamma"].reshape(natom, np1), (1, dup)).reshape(-1)
        out, o = [], 0
        for n in nl["img_ndc"]:
            blk = nl["chi"][o:o + n * np1]
            out += [blk] + [blk * 10.0 ** -(3 * k) for k in range(1, dup)]
            o += n * np1
        nl["chi"] = np.concatenate(out)
    ctx = sg.Context(*N, 6, c, c, c, h ** 3)
    ctx.set_nonlocal(nl["ip_displ"], nl["gamma"], nl["img_atom"], nl["img_ndc"], nl["grid_pos"],
                     nl["chi"])
    return ctx, Oracle(grid, nl), rng, nl


@pytest.mark.parametrize("natom,rc,lmax,dup", [(1, 1.3, 0, 1), (5, 2.0, 2, 1), (6, 2.2, 2, 2),
                                               (9, 4.5, 2, 1), (24, 4.5, 2, 2)])
def test_nonlocal_products(gpu_available, natom, rc, lmax, dup):
    """One projector, 9, 18 (the second half a thousandth of the first), spheres that wrap and
    overlap, and more rows over a point than the fixed-point sums hold (the FP64 kernels stay);
    column counts around the group of 32 and over columns of very different size. The error of a
    column is at most that of the two FP64 contractions: n 2^-53 times the products' magnitudes,
    with n the points of a sphere plus the rows over a point."""
    N, h = (21, 18, 26), 0.45
    ctx, o, rng, nl = _nonlocal_case(N, h, natom, rc, lmax, 3 + natom, dup)
    Nd = N[0] * N[1] * N[2]
    absnl = dict(nl, chi=np.abs(nl["chi"]), gamma=np.abs(nl["gamma"]))
    oabs = Oracle(dict(Nx=N[0], Ny=N[1], Nz=N[2], FDn=6, cx=np.zeros(7), cy=np.zeros(7),
                       cz=np.zeros(7), dV=h ** 3), absnl)
    rows = np.bincount(nl["grid_pos"], minlength=Nd).max() * (lmax + 1) ** 2 * dup
    n = nl["img_ndc"].max() + rows
    for ncol in (1, 31, 33, 70):
        x = rng.uniform(-1, 1, (ncol, Nd)) * 10.0 ** rng.uniform(-6, 6, (ncol, 1))
        y = np.zeros_like(x)
        ctx.Vnl_vec_mult(x, y)
        ref = o.vnl(x)
        size = oabs.vnl(np.abs(x)).max(axis=1)
        assert np.all(np.abs(y - ref).max(axis=1) <= n * 2.0 ** -53 * size), ncol
        if rows <= 128:  # the fixed-point form adds in a fixed order (the FP64 one by atomics)
            y2 = np.zeros_like(x)
            ctx.Vnl_vec_mult(x, y2)
            assert np.array_equal(y, y2)
    ctx.close()


def test_nonlocal_nonfinite_columns(gpu_available):
    """NaN, infinities and extreme exponents stay in their own columns."""
    N, h = (21, 18, 26), 0.45
    ctx, o, rng, _ = _nonlocal_case(N, h, 6, 2.4, 2, 11)
    Nd = N[0] * N[1] * N[2]
    x = rng.uniform(-1, 1, (40, Nd))
    ref = o.vnl(x)
    x[3] *= 1e-300
    x[5, :] = np.nan
    x[7, ::5] = np.inf
    x[33] *= 1e290
    x[36] = 0.0
    y = np.zeros_like(x)
    ctx.Vnl_vec_mult(x, y)
    keep = [i for i in range(40) if i not in (3, 5, 7, 33, 36)]
    big = np.abs(ref).max()
    assert np.abs(y[keep] - ref[keep]).max() <= 1e-12 * big
    assert np.abs(y[3] * 1e300 - ref[3]).max() <= 1e-12 * big
    assert np.abs(y[33] * 1e-290 - ref[33]).max() <= 1e-12 * big
    covered = np.abs(ref[0]) > 0
    assert np.all(np.isnan(y[5][covered])) and not np.any(np.isfinite(y[7][covered]))
    assert np.all(y[36] == 0.0) and np.all(y[:, ~covered] == 0.0)
    ctx.close()


def _kpt_case(N, h, natom, seed):
    rng = np.random.default_rng(seed)
    c = fd_d2_coeffs(6, h)
    grid = dict(Nx=N[0], Ny=N[1], Nz=N[2], FDn=6, cx=c, cy=c, cz=c, dV=h ** 3)
    nl = synthetic_nonlocal(rng, N, h, natom=natom, rc=1.6)
    L = np.array(N) * h
    # two images per atom at most matter here: give every image a copy of the cell
    coords = rng.uniform(0, 1, (len(nl["img_atom"]), 3)) * L + rng.integers(-1, 2, (len(nl["img_atom"]), 3)) * L
    ctx = sg.Context(*N, 6, c, c, c, h ** 3)
    v = rng.normal(size=N[0] * N[1] * N[2])
    ctx.set_veff(np.concatenate([v, -0.5 * v]), nspin=2)
    ctx.set_nonlocal(nl["ip_displ"], nl["gamma"], nl["img_atom"], nl["img_ndc"], nl["grid_pos"],
                     nl["chi"])
    ctx.set_kpoint_geometry(L, coords)
    S = 1.5 * (abs(c[0]) + 2 * np.abs(c[1:]).sum()) + np.abs(v).max()
    return ctx, Oracle(grid, nl), rng, L, coords, v, S


@pytest.mark.parametrize("N", [(17, 14, 20), (6, 12, 9), (34, 13, 12), (25, 24, 31)])
def test_bloch_columns(gpu_available, N):
    """Tiles with halos across the cell faces, Bloch vectors with zero, half and other components,
    column counts around the group of 16, both spins, one block and batched, a non-finite column.
    One apply is off by at most the oracle's own rounding: 80 units of 2^-53 (complex factors
    double the real kernel's 40) of the sum of coefficients, plus as much for the projectors."""
    import torch
    ctx, o, rng, L, co, v, S = _kpt_case(N, 0.45, 3, sum(N))
    Nd = N[0] * N[1] * N[2]
    ks = [2 * np.pi / L * np.array(q) for q in ((0, 0, 0), (0.5, 0, -0.25), (0.1, 0.3, 0.2))]
    for k in ks:
        for ncol in (1, 15, 17):
            x = rng.uniform(-1, 1, (ncol, Nd)) + 1j * rng.uniform(-1, 1, (ncol, Nd))
            y = np.zeros_like(x)
            ctx.Hamiltonian_vectors_mult_kpt(k, -7.0, x, y, spin=1)
            ref = o.hamiltonian_kpt(k, L, co, -0.5 * v, -7.0, x)
            vnl = np.abs(o.vnl_kpt(k, L, co, x)).max()
            assert np.abs(y - ref).max() <= 80 * 2.0 ** -53 * (1.5 * (S + 7.0) + 200 * vnl)
    blocks, x0 = [], []
    for i, k in enumerate(ks):
        for spin in (0, 1):
            ncol = (3, 16, 20)[i]
            x = torch.complex(torch.from_numpy(rng.uniform(-1, 1, (ncol, Nd))),
                              torch.from_numpy(rng.uniform(-1, 1, (ncol, Nd)))).cuda()
            if i == 1 and spin == 0:
                x[4, 7] = float("nan")
            x0.append(x.clone())
            blocks.append(dict(spin=spin, k=[float(q) for q in k], X=x, Y=torch.empty_like(x),
                               a=0.3 * S, b=2.5 * S, a0=-2.0 * S))
    for rep in range(2):  # the second call replays the captured launches on new numbers
        for b, x in zip(blocks, x0):
            b["X"].copy_(x)
        ctx.ChebyshevFiltering_batched(blocks, 5)
        for i, (b, x) in enumerate(zip(blocks, x0)):
            X, Y = x.cpu().numpy().copy(), np.zeros((x.shape[0], Nd), dtype=np.complex128)
            ctx.ChebyshevFiltering_kpt(np.array(b["k"]), X, Y, 5, b["a"], b["b"], b["a0"],
                                       spin=b["spin"])
            y, xx = b["Y"].cpu().numpy(), b["X"].cpu().numpy()
            ok = [n for n in range(x.shape[0]) if not (i == 2 and n == 4)]
            assert np.isfinite(y[ok]).all()
            assert np.abs(y - Y)[ok].max() <= 1e-12 * np.abs(Y[ok]).max()
            assert np.abs(xx - X)[ok].max() <= 1e-12 * np.abs(X[ok]).max()
            if i == 2:
                assert np.isnan(y[4]).any()
        if rep == 0:
            for b in blocks:  # other bounds: the same shapes and buffers
                b["b"] *= 1.1
    ctx.close()


def test_bloch_blocks_of_uneven_widths(gpu_available):
    """One column beside many: most thread blocks of the narrow member have no column group. Every
    column is the one of the single call to the rounding of four degrees."""
    import torch
    ctx, o, rng, L, co, v, S = _kpt_case((17, 14, 20), 0.45, 3, 8)
    Nd = 17 * 14 * 20
    k = 2 * np.pi / L * np.array((0.1, 0.3, 0.2))
    xs = [torch.complex(torch.from_numpy(rng.uniform(-1, 1, (n, Nd))),
                        torch.from_numpy(rng.uniform(-1, 1, (n, Nd)))) for n in (1, 90, 17, 2)]
    blocks = [dict(spin=0, k=[float(q) for q in k], X=x.cuda(), Y=torch.empty_like(x, device="cuda"),
                   a=0.3 * S, b=2.5 * S, a0=-2.0 * S) for x in xs]
    ctx.ChebyshevFiltering_batched(blocks, 4)
    for b, x in zip(blocks, xs):
        X, Y = x.numpy().copy(), np.zeros(x.shape, dtype=np.complex128)
        ctx.ChebyshevFiltering_kpt(k, X, Y, 4, b["a"], b["b"], b["a0"])
        assert np.abs(b["Y"].cpu().numpy() - Y).max() <= 1e-12 * np.abs(Y).max()
    ctx.close()


@pytest.mark.parametrize("ncol", [1, 40])
@pytest.mark.parametrize("N", [(17, 14, 20), (6, 12, 9), (34, 13, 12), (25, 24, 31), (41, 7, 6)])
def test_complex64_tiles(gpu_available, N, ncol):
    """Two degrees of the complex64 filter against complex128. Bound: 40 units of 2^-24 (37 terms in
    chains of six, the factor and the roundings of values and weights take fewer) of the sum of
    |coefficient| times the largest value, for each application."""
    h, a, b, a0 = 0.4, 0.5, 40.0, -0.8
    rng = np.random.default_rng(sum(N) + ncol)
    c = fd_d2_coeffs(6, h)
    ctx = sg.Context(*N, 6, c, c, c, h ** 3)
    Nd = N[0] * N[1] * N[2]
    v = rng.normal(size=Nd)
    ctx.set_veff(v)
    L = np.array(N) * h
    ctx.set_kpoint_geometry(L, np.zeros((0, 3)))
    x = rng.uniform(-1, 1, (ncol, Nd)) + 1j * rng.uniform(-1, 1, (ncol, Nd))
    e, cen = 0.5 * (b - a), 0.5 * (b + a)
    s1 = e / (a0 - cen)
    s2 = 1.0 / (2.0 / s1 - s1)
    S = 1.5 * (abs(c[0]) + 2 * np.abs(c[1:]).sum()) + np.abs(v).max() + cen
    u = 40 * 2.0 ** -24 * np.sqrt(2.0)
    for k in ((0.0, 0.0, 0.0), (0.0, np.pi / L[1], 0.0), (0.3, -0.2, 0.1)):
        y, ref = np.zeros_like(x), np.zeros_like(x)
        ctx.ChebyshevFiltering_kpt(list(k), x.copy(), y, 2, a, b, a0, precision=sg.SGPU_PREC_FP32)
        ctx.ChebyshevFiltering_kpt(list(k), x.copy(), ref, 2, a, b, a0)
        m0 = np.sqrt(2.0)
        m1 = abs(s1 / e) * S * m0                      # bound of the first iterate
        e1 = u * m1
        e2 = abs(2 * s2 / e) * S * (e1 + u * m1) + 3 * 2.0 ** -24 * abs(s1 * s2) * m0
        assert np.abs(y - ref).max() <= e2, k
    # an infinity spreads as it does in the general kernel
    x[0, Nd // 2] = np.inf
    x[-1, 3] = np.nan
    out = []
    for on in (True, False):
        ctx.set_zstencil_pairs(on)
        y = np.zeros_like(x)
        ctx.ChebyshevFiltering_kpt([0.3, -0.2, 0.1], x.copy(), y, 2, a, b, a0,
                                   precision=sg.SGPU_PREC_FP32)
        out.append(np.isfinite(y))
    assert np.array_equal(out[0], out[1])
    ctx.close()


def test_filter_against_extended_precision(gpu_available):
    """What repeats in every application (rounded coefficients, values cut one way) adds up over the
    degrees of a filter: one column of a degree-20 filter, in norm, within two roundings of 2^-53."""
    N, h, m, a, b, a0 = (26, 22, 31), 0.4, 20, 0.5, 50.0, -1.0
    rng = np.random.default_rng(11)
    c = fd_d2_coeffs(6, h)
    ctx = sg.Context(*N, 6, c, c, c, h ** 3)
    Nd = N[0] * N[1] * N[2]
    v = rng.normal(size=Nd)
    ctx.set_veff(v)
    x = rng.uniform(-1, 1, (6, Nd))
    y = np.zeros_like(x)
    ctx.ChebyshevFiltering(x.copy(), y, m, a, b, a0)
    ctx.close()
    ld = np.longdouble
    e, cen = 0.5 * (b - a), 0.5 * (b + a)
    c0 = (c[0] * -0.5 + c[0] * -0.5) + c[0] * -0.5 - cen  # the scalars as doubles
    shape = N[::-1]

    def apply(u):
        r = (ld(c0) + v.astype(ld).reshape(shape)) * u
        for ax in range(3):
            for q in range(1, 7):
                r = r + ld(c[q] * -0.5) * (np.roll(u, q, ax) + np.roll(u, -q, ax))
        return r

    sigma = e / (a0 - cen)
    gamma = 2.0 / sigma
    prev = x[0].astype(ld).reshape(shape)
    cur = apply(prev) * ld(sigma / e)
    for _ in range(1, m):
        s2 = 1.0 / (gamma - sigma)
        prev, cur = cur, apply(cur) * ld(2.0 * s2 / e) - ld(sigma * s2) * prev
        sigma = s2
    cur = cur.reshape(-1)
    err = np.sqrt(((y[0] - cur) ** 2).sum() / (cur ** 2).sum())
    assert err <= 2 * 2.0 ** -53


def test_filter_of_columns_around_a_point(gpu_available):
    """Columns that fall off by exp(-0.9 r) (Bohr) from a point, filters of degree 20 up to the end of
    the spectrum: the fixed-point kernels' error against extended precision, over eight columns, is
    at most three quarters of the FP64 kernels' (half of it; ties rounded to one side: 0.85)."""
    N, h, m, a, a0 = (26, 22, 24), 0.39, 20, 0.5, -1.0
    rng = np.random.default_rng(12)
    c = fd_d2_coeffs(6, h)
    ctx = sg.Context(*N, 6, c, c, c, h ** 3)
    Nd, ncol = N[0] * N[1] * N[2], 8
    v = rng.normal(0.0, 0.7, Nd)
    ctx.set_veff(v)
    b = -1.5 * (c[0] + 2 * sum((-1) ** q * c[q] for q in range(1, 7))) + v.max()
    g = np.meshgrid(*[np.arange(n) / n for n in N[::-1]], indexing="ij")
    x = np.zeros((ncol, Nd))
    for n in range(ncol):
        u = sum(rng.normal() * np.cos(2 * np.pi * (sum(q * w for q, w in zip(rng.integers(-2, 3, 3), g))
                                                   + rng.uniform())) for _ in range(4))
        p = rng.uniform(0, 1, 3)
        d2 = sum((np.minimum(abs(w - s), 1 - abs(w - s)) * k * h) ** 2 for w, s, k in zip(g, p, N[::-1]))
        x[n] = (u * np.exp(-0.9 * np.sqrt(d2 + 0.5))).reshape(-1)
    got = {}
    for on in (True, False):
        ctx.set_fixed_point(on)
        y = np.zeros_like(x)
        ctx.ChebyshevFiltering(x.copy(), y, m, a, b, a0)
        got[on] = y
    ctx.close()
    ld = np.longdouble
    e, cen = 0.5 * (b - a), 0.5 * (b + a)
    c0 = (c[0] * -0.5 + c[0] * -0.5) + c[0] * -0.5 - cen
    shape = (ncol,) + N[::-1]

    def apply(u):
        r = (ld(c0) + v.astype(ld).reshape(shape[1:])) * u
        for ax in (1, 2, 3):
            for q in range(1, 7):
                r = r + ld(c[q] * -0.5) * (np.roll(u, q, ax) + np.roll(u, -q, ax))
        return r

    sigma = e / (a0 - cen)
    gamma = 2.0 / sigma
    prev = x.astype(ld).reshape(shape)
    cur = apply(prev) * ld(sigma / e)
    for _ in range(1, m):
        s2 = 1.0 / (gamma - sigma)
        prev, cur = cur, apply(cur) * ld(2.0 * s2 / e) - ld(sigma * s2) * prev
        sigma = s2
    cur = cur.reshape(ncol, Nd)
    size = np.sqrt((cur ** 2).sum(axis=1))
    err = {on: float(np.sqrt((((got[on] - cur) ** 2).sum(axis=1) / size ** 2).mean())) for on in got}
    assert err[True] <= 0.75 * err[False]


@pytest.mark.parametrize("bloch", [False, True])
@pytest.mark.parametrize("vmax", [0.0, 31.0])
def test_roundings_have_no_preferred_side(gpu_available, vmax, bloch):
    """Values that all lie halfway between two fixed-point numbers (2^-5 of their blocks' largest, an
    odd last bit), with and without a potential whose products end in half a unit every other time: the
    mean error over 300000 points is at most a tenth of the shift times the quantum, 2^-56, where ties
    rounded to one side leave 0.6 of it (with the potential 1.1)."""
    N, h, ncol, shift = (32, 30, 40), 0.4, 8, 25.0
    rng = np.random.default_rng(4)
    c = fd_d2_coeffs(6, h)
    Nd = N[0] * N[1] * N[2]
    ctx = sg.Context(*N, 6, c, c, c, h ** 3)
    x = (1.0 + (2 * rng.integers(0, 2 ** 51, (ncol, Nd)) + 1) * 2.0 ** -52) * 2.0 ** -5
    z, r = np.divmod(np.arange(Nd), N[0] * N[1])
    y_, x_ = np.divmod(r, N[0])
    peak = (z % 6 == 1) & (y_ % 5 == 2) & (x_ % 8 == 3)  # one in every tile's window
    x[:, peak] = 1.0
    v = rng.uniform(17.0, vmax, Nd) if vmax else np.zeros(Nd)
    ld = np.longdouble
    c0 = (c[0] * -0.5 + c[0] * -0.5) + c[0] * -0.5 + shift
    u = x.astype(ld).reshape((ncol,) + N[::-1])
    ref = (ld(c0) + v.astype(ld).reshape(N[::-1])) * u
    for ax in (1, 2, 3):
        for q in range(1, 7):
            ref = ref + ld(c[q] * -0.5) * (np.roll(u, q, ax) + np.roll(u, -q, ax))
    ref = ref.reshape(ncol, Nd)
    if bloch:
        ctx.set_kpoint_geometry(np.array(N) * h, np.zeros((0, 3)))
        y = np.zeros((ncol, Nd), dtype=complex)
        ctx.Lap_plus_diag_vec_mult_orth_kpt(np.zeros(3), -0.5, 1.0, shift, v, x + 1j * x, y)
        err = [y.real - ref, y.imag - ref]
    else:
        y = np.zeros_like(x)
        ctx.Lap_plus_diag_vec_mult_orth(-0.5, 1.0, shift, v, x, y)
        err = [y - ref]
    ctx.close()
    for e in err:
        assert abs(float(e[:, ~peak].mean())) <= 0.1 * shift * 2.0 ** -56
