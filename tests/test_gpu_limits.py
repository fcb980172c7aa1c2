"""What a call does when device scratch, a table or a kernel's bounded wait fails (failures made on
the host, sgpu_inject_failure), and at the edges of what the fixed-point FP64 kernels take."""
import ctypes

import numpy as np
import pytest

import sparc_gb300 as sg
from oracle.oracle import Oracle
from sparc_gb300.synthetic import fd_d2_coeffs, synthetic_nonlocal

pytestmark = pytest.mark.gpu

SCRATCH, TABLES, RR_WAIT, SMALL, FIRST_TRY = 1, 2, 4, 8, 16


def _system(N, h, natom=6, rc=2.2, nspin=1, seed=1):
    """A context with a potential and projectors, and the arrays they were made from."""
    rng = np.random.default_rng(seed)
    c = fd_d2_coeffs(6, h)
    Nd = N[0] * N[1] * N[2]
    nl = synthetic_nonlocal(rng, N, h, natom=natom, rc=rc) if natom else None
    ctx = sg.Context(*N, 6, c, c, c, h ** 3)
    v = rng.normal(0.0, 0.4, nspin * Nd)
    _set(ctx, v, nl, nspin)
    return ctx, v, nl, dict(Nx=N[0], Ny=N[1], Nz=N[2], FDn=6, cx=c, cy=c, cz=c, dV=h ** 3), rng


def _set(ctx, v, nl, nspin=1):
    ctx.set_veff(v, nspin=nspin)
    if nl:
        ctx.set_nonlocal(nl["ip_displ"], nl["gamma"], nl["img_atom"], nl["img_ndc"],
                         nl["grid_pos"], nl["chi"])


def _close(a, b, tol=1e-12):
    """Equal to the rounding of two FP64 routes, relative to the largest value."""
    assert np.isfinite(b).all()
    assert np.abs(a - b).max() <= tol * np.abs(b).max()


def test_failed_allocation_is_not_met_again(gpu_available):
    """A block that no device holds is refused for want of memory; the next call is not affected by
    the allocation that failed."""
    N, h = (30, 28, 26), 0.4
    ctx, v, nl, grid, rng = _system(N, h)
    Nd = ctx.Nd
    x = rng.uniform(-1, 1, (8, Nd))
    y = np.zeros_like(x)
    rc = sg.lib().sgpu_Lap_vec_mult(ctx._h, 2 ** 31 - 1, ctypes.c_double(0.1), sg._ptr(x), Nd,
                                    sg._ptr(y), Nd)
    assert rc == 3, sg.lib().sgpu_last_error().decode()
    ctx.Lap_vec_mult(0.1, x, y)
    _close(y, Oracle(grid, None).lap_plus_diag(1.0, 0.0, 0.1, None, x))
    ctx.close()


def test_rr_products_without_scratch(gpu_available):
    """No room for the slices: the FP64 GEMMs."""
    ctx, v, nl, grid, rng = _system((30, 28, 26), 0.4, natom=0)
    ncol = 70
    Y = rng.uniform(-1, 1, (ncol, ctx.Nd))
    Q = rng.normal(size=(ncol, ncol))
    ctx.inject_failure(SCRATCH)
    HY, Hp, Mp, X = np.zeros_like(Y), np.zeros_like(Q), np.zeros_like(Q), np.zeros_like(Y)
    ctx.Project_Hamiltonian(Y, HY, Hp, Mp)
    ctx.Subspace_Rotation(Y, Q, X)
    _close(Mp, Y @ Y.T)
    _close(Hp, Y @ HY.T)
    _close(X, Q @ Y)
    ctx.close()


@pytest.mark.parametrize("ncol", [7, 70])
def test_rr_products_after_a_wait_ran_out(gpu_available, ncol):
    """A block that gave up a wait leaves tiles unwritten: the products are formed again by the FP64
    GEMMs, and nothing is left in the status word."""
    ctx, v, nl, grid, rng = _system((30, 28, 26), 0.4, natom=0)
    Y = rng.uniform(-1, 1, (ncol, ctx.Nd))
    Q = rng.normal(size=(ncol, ncol))
    ctx.inject_failure(RR_WAIT)
    HY, Hp, Mp, X = np.zeros_like(Y), np.zeros_like(Q), np.zeros_like(Q), np.zeros_like(Y)
    ctx.Project_Hamiltonian(Y, HY, Hp, Mp)
    ctx.Subspace_Rotation(Y, Q, X)
    _close(Mp, Y @ Y.T)
    _close(Hp, Y @ HY.T)
    _close(X, Q @ Y)
    ctx.inject_failure(0)
    assert ctx.kernel_status() == 0
    ctx.close()


def test_smallest_coefficients_and_values(gpu_available):
    """Coefficients that add up to 2e-60 and values of 1.5e-231 beside others 2^-55 of it: results
    down to the smallest exponents, within the bound of the 37-term sum."""
    N, h = (50, 48, 46), 0.4
    Nd = N[0] * N[1] * N[2]
    c = fd_d2_coeffs(6, h)
    S0 = 3 * (abs(c[0]) + 2 * np.abs(c[1:]).sum())
    c = c * (2e-60 / S0)
    ctx = sg.Context(*N, 6, c, c, c, h ** 3)
    grid = dict(Nx=N[0], Ny=N[1], Nz=N[2], FDn=6, cx=c, cy=c, cz=c, dV=h ** 3)
    rng = np.random.default_rng(3)
    x = rng.choice([-1.0, 1.0], size=(1, Nd)) * 1.5e-231 * 2.0 ** -55
    x[0, rng.integers(0, Nd, 200)] = 1.5e-231
    y = np.zeros_like(x)
    ctx.Lap_vec_mult(0.0, x, y)
    ref = Oracle(grid, None).lap_plus_diag(1.0, 0.0, 0.0, None, x)
    assert np.isfinite(y).all()
    assert np.abs(y - ref).max() <= 40 * 2.0 ** -53 * 2e-60 * 1.5e-231 + 40 * 5e-324
    ctx.close()


def test_more_projector_rows_than_a_grid_dimension(gpu_available):
    """7300 atoms of nine projectors, five points each: 65700 rows, real and complex."""
    import torch
    N, h, natom, npt = (40, 40, 40), 0.4, 7300, 5
    Nd = N[0] * N[1] * N[2]
    rng = np.random.default_rng(2)
    nl = dict(ip_displ=np.arange(natom + 1, dtype=np.int32) * 9,
              gamma=rng.uniform(-2, 2, 9 * natom), img_atom=np.arange(natom, dtype=np.int32),
              img_ndc=np.full(natom, npt, dtype=np.int32),
              grid_pos=np.concatenate([np.sort(rng.choice(Nd, npt, replace=False))
                                       for _ in range(natom)]).astype(np.int32),
              chi=rng.uniform(-1, 1, 9 * npt * natom))
    c = fd_d2_coeffs(6, h)
    grid = dict(Nx=N[0], Ny=N[1], Nz=N[2], FDn=6, cx=c, cy=c, cz=c, dV=h ** 3)
    ctx = sg.Context(*N, 6, c, c, c, h ** 3)
    v = rng.normal(0.0, 0.4, Nd)
    _set(ctx, v, nl)
    L = np.array(N) * h
    coords = rng.uniform(0, 1, (natom, 3)) * L
    ctx.set_kpoint_geometry(L, coords)
    o = Oracle(grid, nl)
    x = rng.uniform(-1, 1, (3, Nd))
    y = np.zeros_like(x)
    ctx.Vnl_vec_mult(x, y)
    _close(y, o.vnl(x))
    z = x + 1j * rng.uniform(-1, 1, (3, Nd))
    k = np.array([0.2, -0.1, 0.3])
    w = np.zeros_like(z)
    ctx.Vnl_vec_mult_kpt(k, z, w)
    _close(w, o.vnl_kpt(k, L, coords, z))
    X = torch.from_numpy(z).cuda()
    Y = torch.empty_like(X)
    ctx.ChebyshevFiltering_batched([dict(spin=0, k=k, X=X, Y=Y, a=0.5, b=40.0, a0=-0.8)], 2)
    _close(Y.cpu().numpy(), o.chebyshev_kpt(k, L, coords, v, 2, 0.5, 40.0, -0.8, z)[1])
    ctx.close()


def test_nonlocal_and_stencil_without_scratch(gpu_available):
    """No room for the partial projections or a caller's potential as digits: the FP64 kernels, in
    every call that uses either, real and complex, single and batched. Room for some column groups'
    partial projections: those take turns."""
    import torch
    N, h = (30, 28, 26), 0.4
    ctx, v, nl, grid, rng = _system(N, h)
    o, Nd, ncol = Oracle(grid, nl), ctx.Nd, 165
    L = np.array(N) * h
    coords = rng.uniform(0, 1, (len(nl["img_atom"]), 3)) * L
    ctx.set_kpoint_geometry(L, coords)
    x = rng.uniform(-1, 1, (ncol, Nd))
    z = x[:90] + 1j * rng.uniform(-1, 1, (90, Nd))
    k = np.array([0.2, -0.1, 0.3])
    zt = torch.from_numpy(z).cuda()
    for mask in (SCRATCH, SMALL, 0):
        ctx.inject_failure(mask)
        y = np.zeros_like(x)
        ctx.Vnl_vec_mult(x, y)
        _close(y, o.vnl(x))
        ctx.Lap_plus_diag_vec_mult_orth(-0.5, 1.0, 0.3, v, x, y)
        _close(y, o.lap_plus_diag(-0.5, 1.0, 0.3, v, x))
        ctx.Hamiltonian_vectors_mult(0.3, x, y)
        _close(y, o.hamiltonian(v, 0.3, x))
        X, Y = x.copy(), np.zeros_like(x)
        ctx.ChebyshevFiltering(X, Y, 5, 0.5, 40.0, -0.8)
        Xo, Yo = o.chebyshev(v, 5, 0.5, 40.0, -0.8, x)
        _close(Y, Yo)
        _close(X, Xo)
        w = np.zeros_like(z)
        ctx.Hamiltonian_vectors_mult_kpt(k, 0.3, z, w)
        _close(w, o.hamiltonian_kpt(k, L, coords, v, 0.3, z))
        Xo, Yo = o.chebyshev_kpt(k, L, coords, v, 5, 0.5, 40.0, -0.8, z)
        cuts = [0, 3, 40, 41, 90]
        blocks = [dict(spin=0, k=k, X=zt[i:j].clone(), Y=torch.empty_like(zt[i:j]), a=0.5, b=40.0,
                       a0=-0.8) for i, j in zip(cuts, cuts[1:])]
        ctx.ChebyshevFiltering_batched(blocks, 5)
        for blk, i, j in zip(blocks, cuts, cuts[1:]):
            _close(blk["Y"].cpu().numpy(), Yo[i:j])
            _close(blk["X"].cpu().numpy(), Xo[i:j])
    ctx.close()


def test_sets_without_tables(gpu_available):
    """No room for the fixed-point tables of the potential or the projectors: both sets are accepted
    as before and the FP64 kernels serve them; a later set has its tables again."""
    import torch
    N, h = (30, 28, 26), 0.4
    ctx, v, nl, grid, rng = _system(N, h)
    o, Nd, ncol = Oracle(grid, nl), ctx.Nd, 11
    L = np.array(N) * h
    coords = rng.uniform(0, 1, (len(nl["img_atom"]), 3)) * L
    ctx.set_kpoint_geometry(L, coords)
    x = rng.uniform(-1, 1, (ncol, Nd))
    z = x + 1j * rng.uniform(-1, 1, (ncol, Nd))
    k = np.array([0.2, -0.1, 0.3])
    zt = torch.from_numpy(z).cuda()
    for mask in (TABLES, 0):
        ctx.inject_failure(mask)
        _set(ctx, np.concatenate([v, -0.5 * v]), nl, 2)
        for spin, s in ((0, 1.0), (1, -0.5)):
            y = np.zeros_like(x)
            ctx.Hamiltonian_vectors_mult(0.3, x, y, spin=spin)
            _close(y, o.hamiltonian(s * v, 0.3, x))
            X, Y = x.copy(), np.zeros_like(x)
            ctx.ChebyshevFiltering(X, Y, 4, 0.5, 40.0, -0.8, spin=spin)
            _close(Y, o.chebyshev(s * v, 4, 0.5, 40.0, -0.8, x)[1])
            w = np.zeros_like(z)
            ctx.Hamiltonian_vectors_mult_kpt(k, 0.3, z, w, spin=spin)
            _close(w, o.hamiltonian_kpt(k, L, coords, s * v, 0.3, z))
            Xb, Yb = zt.clone(), torch.empty_like(zt)
            ctx.ChebyshevFiltering_batched([dict(spin=spin, k=k, X=Xb, Y=Yb, a=0.5, b=40.0,
                                                 a0=-0.8)], 4)
            _close(Yb.cpu().numpy(), o.chebyshev_kpt(k, L, coords, s * v, 4, 0.5, 40.0, -0.8, z)[1])
        _set(ctx, v, nl, 1)
    ctx.close()


def test_rr_products_in_many_passes(gpu_available):
    """Slices held to 1 MB: 43 ranges of 512 points, whose sums take no more room than one range's."""
    import torch
    N, ncol = (30, 28, 26), 200
    ctx, v, nl, grid, rng = _system(N, 0.4, natom=0)
    Y = torch.from_numpy(rng.uniform(-1, 1, (ncol, ctx.Nd))).cuda()
    Q = torch.from_numpy(rng.normal(size=(ncol, ncol))).cuda()
    HY, X, Hp, Mp = torch.empty_like(Y), torch.empty_like(Y), torch.empty_like(Q), torch.empty_like(Q)
    ctx.inject_failure(SMALL)
    ctx.Project_Hamiltonian(Y[:64], HY[:64], Hp[:64, :64].contiguous(), Mp[:64, :64].contiguous())
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    ctx.Project_Hamiltonian(Y, HY, Hp, Mp)
    ctx.Subspace_Rotation(Y, Q, X)
    torch.cuda.synchronize()
    # two operands of 2 MB (the least range), one set of 200 x 200 sums, an eighth of slack each
    assert free - torch.cuda.mem_get_info()[0] < 16 << 20
    y, hy = Y.cpu().numpy(), HY.cpu().numpy()
    _close(Mp.cpu().numpy(), y @ y.T)
    _close(Hp.cpu().numpy(), y @ hy.T)
    _close(X.cpu().numpy(), Q.cpu().numpy() @ y)
    ctx.close()


@pytest.mark.parametrize("N", [(18, 14, 170), (33, 30, 130)])
@pytest.mark.parametrize("ncol", [4, 300])
@pytest.mark.parametrize("bloch", [False, True])
def test_columns_that_decay(gpu_available, N, ncol, bloch):
    """A slab's states fall off into the vacuum, here by exp(-0.35) a plane and by 1e-10 and more in
    all, and rise again behind it. A block's scale is below 2^5 of the largest value that it loaded in
    its last 14 steps, planes at most 14 away, and values are rounded to 2^-57 of the scale: a
    result is off by at most 40 units of 2^-53 of the sum of |coefficient| (as many again for the
    parts of a complex value) times the largest value of the planes up to 16 away."""
    h, dz = 0.4, 16
    rng = np.random.default_rng(sum(N) + ncol)
    c = fd_d2_coeffs(6, h)
    Nd, per = N[0] * N[1] * N[2], N[0] * N[1]
    ctx = sg.Context(*N, 6, c, c, c, h ** 3)
    z = np.arange(N[2])
    d = np.minimum((z - 20) % N[2], (20 - z) % N[2])
    prof = np.exp(-0.35 * d)
    some = rng.choice(ncol, 3)
    x = rng.uniform(-1, 1, (ncol, Nd)) * np.repeat(prof, per)
    S = 1.5 * (abs(c[0]) + 2 * np.abs(c[1:]).sum()) + 0.7
    near = np.max([np.roll(prof, s) for s in range(-dz, dz + 1)], axis=0)
    tol = 40 * 2.0 ** -53 * S * np.repeat(near, per)
    ld = np.longdouble
    if bloch:
        ctx.set_kpoint_geometry(np.array(N) * h, np.zeros((0, 3)))
        x = x + 1j * rng.uniform(-1, 1, (ncol, Nd)) * np.repeat(prof, per)
        y = np.zeros_like(x)
        ctx.Lap_plus_diag_vec_mult_orth_kpt(np.zeros(3), -0.5, 0.0, 0.7, None, x, y)
        tol = 2 * tol
    else:
        y = np.zeros_like(x)
        ctx.Lap_plus_diag_vec_mult_orth(-0.5, 0.0, 0.7, None, x, y)
    for n in some:
        u = x[n].reshape(N[::-1]).astype(np.clongdouble if bloch else ld)
        r = (ld(-0.5) * 3 * ld(c[0]) + ld(0.7)) * u
        for ax in range(3):
            for q in range(1, 7):
                r = r + ld(-0.5) * ld(c[q]) * (np.roll(u, q, ax) + np.roll(u, -q, ax))
        assert np.all(np.abs(y[n] - r.reshape(-1)) <= tol)
    ctx.close()


@pytest.mark.parametrize("ncol", [3, 300])
def test_fp64_arithmetic_on_request(gpu_available, ncol):
    """set_fixed_point(False): every point is as accurate as the values that its own stencil or
    projectors touch, 40 units of 2^-53 of the sum of |coefficient| times the largest value of six
    planes around, and n units of the products' magnitudes at the point itself (n: points of a
    sphere and rows over a point). Columns fall off along z."""
    N, h = (18, 14, 90), 0.4
    ctx, v, nl, grid, rng = _system(N, h, natom=7, rc=2.2)
    ctx.set_fixed_point(False)
    Nd, per, c = ctx.Nd, N[0] * N[1], grid["cx"]
    z = np.arange(N[2])
    prof = np.exp(-0.35 * np.minimum((z - 20) % N[2], (20 - z) % N[2]))
    near = np.repeat(np.max([np.roll(prof, s) for s in range(-6, 7)], axis=0), per)
    x = rng.uniform(-1, 1, (ncol, Nd)) * np.repeat(prof, per)
    S = 1.5 * (abs(c[0]) + 2 * np.abs(c[1:]).sum()) + 0.7
    y = np.zeros_like(x)
    ctx.Lap_plus_diag_vec_mult_orth(-0.5, 0.0, 0.7, None, x, y)
    some = rng.choice(ncol, 2)
    lap = Oracle(grid, None).lap_plus_diag(-0.5, 0.0, 0.7, None, x[some])
    assert np.all(np.abs(y[some] - lap) <= 40 * 2.0 ** -53 * S * near)
    ctx.set_kpoint_geometry(np.array(N) * h, np.zeros((len(nl["img_atom"]), 3)))
    w = np.zeros_like(x, dtype=complex)
    ctx.Lap_plus_diag_vec_mult_orth_kpt(np.zeros(3), -0.5, 0.0, 0.7, None, x.astype(complex), w)
    assert np.all(np.abs(w[some] - lap) <= 80 * 2.0 ** -53 * S * near)
    y[:] = 0.0
    ctx.Vnl_vec_mult(x, y)
    size = Oracle(grid, dict(nl, chi=np.abs(nl["chi"]), gamma=np.abs(nl["gamma"]))).vnl(np.abs(x[some]))
    n = nl["img_ndc"].max() + np.bincount(nl["grid_pos"], minlength=Nd).max() * 9
    assert np.all(np.abs(y[some] - Oracle(grid, nl).vnl(x[some])) <= n * 2.0 ** -53 * size)
    with pytest.raises(sg.SgpuError):
        sg._check(sg.lib().sgpu_set_fixed_point(ctx._h, 2))
    ctx.close()


@pytest.mark.parametrize("N", [(47, 14, 12), (96, 9, 12), (64, 13, 7)])
def test_general_complex_kernel_on_wide_planes(gpu_available, N):
    """Planes of 43 points and more along x, where the best tile of the general complex128 stencil
    once had more threads than its blocks may have; alone and batched."""
    import torch
    h = 0.4
    rng = np.random.default_rng(sum(N))
    c = fd_d2_coeffs(6, h)
    Nd, L = N[0] * N[1] * N[2], np.array(N) * h
    ctx = sg.Context(*N, 6, c, c, c, h ** 3)
    v = rng.normal(0.0, 0.4, Nd)
    ctx.set_veff(v)
    ctx.set_kpoint_geometry(L, np.zeros((0, 3)))
    ctx.set_fixed_point(False)
    o = Oracle(dict(Nx=N[0], Ny=N[1], Nz=N[2], FDn=6, cx=c, cy=c, cz=c, dV=h ** 3), None)
    k = np.array([0.2, -0.1, 0.3])
    z = rng.uniform(-1, 1, (3, Nd)) + 1j * rng.uniform(-1, 1, (3, Nd))
    w = np.zeros_like(z)
    ctx.Hamiltonian_vectors_mult_kpt(k, 0.3, z, w)
    _close(w, o.lap_plus_diag_kpt(k, L, -0.5, 1.0, 0.3, v, z))
    X = torch.from_numpy(z).cuda()
    Y = torch.empty_like(X)
    ctx.ChebyshevFiltering_batched([dict(spin=0, k=k, X=X, Y=Y, a=0.5, b=40.0, a0=-0.8)], 4)
    Xf, Yf = z.copy(), np.zeros_like(z)
    ctx.set_fixed_point(True)
    ctx.ChebyshevFiltering_kpt(k, Xf, Yf, 4, 0.5, 40.0, -0.8)
    _close(Y.cpu().numpy(), Yf)
    ctx.close()


def test_two_threads_with_ranges_of_different_size(gpu_available):
    """Two contexts, each used by a thread of its own, whose launches of one kernel ask for different
    amounts of shared memory: neither's calls are disturbed."""
    import threading

    import torch
    work, bad = [], []
    for N, natom, rc in (((24, 22, 20), 1, 1.0), ((30, 28, 26), 30, 3.0)):
        ctx, v, nl, grid, rng = _system(N, 0.4, natom=natom, rc=rc)
        x = torch.from_numpy(rng.uniform(-1, 1, (4, ctx.Nd))).cuda()
        work.append((ctx, x, torch.zeros_like(x), Oracle(grid, nl)))

    def run(ctx, x, y):
        for _ in range(3000):
            try:
                y.zero_()
                ctx.Vnl_vec_mult(x, y)
            except sg.SgpuError as e:
                bad.append(str(e))

    threads = [threading.Thread(target=run, args=w[:3]) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:3]
    for ctx, x, y, o in work:
        _close(y.cpu().numpy(), o.vnl(x.cpu().numpy()))
        ctx.close()


def test_other_allocations_take_scratch_back(gpu_available):
    """Allocations that fail while optional scratch is held (sets, forces, tuning) are tried again
    without it; the calls' results stay."""
    ctx, v, nl, grid, rng = _system((30, 28, 26), 0.4)
    o, cell, ncol = Oracle(grid, nl), np.array((30, 28, 26)) * 0.4, 64
    x = rng.uniform(-1, 1, (ncol, ctx.Nd))
    occ = rng.uniform(0, 1, ncol)
    h, s = np.zeros_like(x), [np.zeros((ncol, ncol)) for _ in range(2)]
    ctx.Project_Hamiltonian(x, h, *s)  # slices and partial projections are kept from here on
    forces = ctx.Calculate_nonlocal_forces(cell, x, occ)
    ctx.Project_Hamiltonian(x, h, *s)
    ctx.inject_failure(FIRST_TRY)
    _close(ctx.Calculate_nonlocal_forces(cell, x, occ), forces, 1e-11)
    ctx.autotune(ncol=16)
    _set(ctx, np.concatenate([v, 0.5 * v]), nl, 2)
    ctx.inject_failure(0)
    y = np.zeros_like(x)
    ctx.Hamiltonian_vectors_mult(0.2, x, y, spin=1)
    _close(y, o.hamiltonian(0.5 * v, 0.2, x))
    ctx.close()


def _padded(x, pad):
    """The rows of x in a device block of longer, poisoned rows."""
    import torch
    b = torch.full((x.shape[0], x.shape[1] + pad), float("nan"), dtype=torch.float64, device="cuda")
    b[:, :x.shape[1]] = torch.from_numpy(x).cuda()
    return b[:, :x.shape[1]]


@pytest.mark.parametrize("ncol,pad", [(5, 1), (33, 7), (70, 64)])
def test_padded_device_blocks(gpu_available, ncol, pad):
    """Leading dimensions above Nd, odd ones among them, in the real FP64 calls above the size of the
    point-per-thread kernel; the second spin of two."""
    N, h = (29, 27, 31), 0.4
    ctx, v, nl, grid, rng = _system(N, h, nspin=2)
    o, Nd = Oracle(grid, nl), ctx.Nd
    v1 = v[Nd:]
    x = rng.uniform(-1, 1, (ncol, Nd))
    X, Y = _padded(x, pad), _padded(np.zeros_like(x), pad)
    assert X.stride(0) == Nd + pad
    ctx.Hamiltonian_vectors_mult(0.3, X, Y, spin=1)
    _close(Y.cpu().numpy(), o.hamiltonian(v1, 0.3, x))
    Y.zero_()
    ctx.Vnl_vec_mult(X, Y)
    _close(Y.cpu().numpy(), o.vnl(x))
    ctx.ChebyshevFiltering(X, Y, 6, 0.5, 40.0, -0.8, spin=1)
    Xo, Yo = o.chebyshev(v1, 6, 0.5, 40.0, -0.8, x)
    _close(Y.cpu().numpy(), Yo)
    _close(X.cpu().numpy(), Xo)
    HY, Z = _padded(np.zeros_like(x), pad), _padded(np.zeros_like(x), pad)
    Hp, Mp = np.zeros((ncol, ncol)), np.zeros((ncol, ncol))
    Q = rng.normal(size=(ncol, ncol))
    ctx.Project_Hamiltonian(Y, HY, Hp, Mp, spin=1)
    ctx.Subspace_Rotation(Y, Q, Z)
    y, hy = Y.cpu().numpy(), HY.cpu().numpy()
    _close(hy, o.hamiltonian(v1, 0.0, y))
    _close(Mp, y @ y.T)
    _close(Hp, y @ hy.T)
    _close(Z.cpu().numpy(), Q @ y)
    for b in (X, Y, HY, Z):  # nothing was written between the columns
        full = b.as_strided((ncol, Nd + pad), (Nd + pad, 1))
        assert np.isnan(full[:, Nd:].cpu().numpy()).all()
    ctx.close()
