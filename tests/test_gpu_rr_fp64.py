"""The plain FP64 Rayleigh-Ritz products on the eight-slice tensor-core kernels (csrc/rr_tc.cu), at
widths around the 64- and 128-column tiles and the step to cuBLAS, and over more grid points than
one workspace pass holds."""
import numpy as np
import pytest

import sparc_gb300 as sg
from sparc_gb300.synthetic import fd_d2_coeffs

pytestmark = pytest.mark.gpu


def _ctx(N):
    c = fd_d2_coeffs(6, 0.4)
    ctx = sg.Context(*N, 6, c, c, c, 0.4 ** 3)
    ctx.set_veff(np.random.default_rng(1).normal(0.0, 0.5, N[0] * N[1] * N[2]))
    return ctx


@pytest.mark.parametrize("ncol", [1, 7, 47, 48, 64, 65, 129, 200])
def test_products_against_extended_precision(gpu_available, ncol):
    """Columns over six decades, one zero. Gram entries: the slices cut a value by at most 2^-57 of
    its column's largest, with random signs, and the result is rounded once: 16 units of 2^-53 of
    |y_m||z_n| covers both (the reference sum is taken in extended precision). Rotation: the same of
    sum |Y||Q| per entry, with the row balance in place of the column norm."""
    N = (16, 14, 13)
    Nd = N[0] * N[1] * N[2]
    rng = np.random.default_rng(ncol)
    ctx = _ctx(N)
    Y = rng.uniform(-1, 1, (ncol, Nd)) * 10.0 ** rng.uniform(-3, 3, (ncol, 1))
    if ncol > 3:
        Y[3] = 0.0
    HY, Hp, Mp = np.zeros_like(Y), np.zeros((ncol, ncol)), np.zeros((ncol, ncol))
    ctx.Project_Hamiltonian(Y, HY, Hp, Mp)
    assert ctx.kernel_status() == 0
    Yl, Hl = Y.astype(np.longdouble), HY.astype(np.longdouble)
    ny, nh = np.linalg.norm(Y, axis=1), np.linalg.norm(HY, axis=1)
    eps = 16 * 2.0 ** -53
    lo = np.tril_indices(ncol)
    some = rng.integers(0, len(lo[0]), size=min(400, len(lo[0])))
    for i, j in zip(lo[0][some], lo[1][some]):
        assert abs(Mp[i, j] - float((Yl[i] * Yl[j]).sum())) <= eps * ny[i] * ny[j]
        assert abs(Hp[i, j] - float((Hl[i] * Yl[j]).sum())) <= eps * nh[i] * ny[j]
    assert np.array_equal(Mp, Mp.T) and np.array_equal(Hp, Hp.T)
    s = np.abs(Y).max(axis=1)
    s[s == 0] = 1.0
    Q = rng.normal(size=(ncol, ncol)) / s[None, :]
    X = np.zeros_like(Y)
    ctx.Subspace_Rotation(Y, Q, X)
    assert ctx.kernel_status() == 0
    rows = rng.integers(0, Nd, size=200)
    ref = (Q.astype(np.longdouble)[:, :, None] * Yl[None, :, rows]).sum(axis=1).astype(np.float64)
    # a grid point's values and a column of Q each have their own scale
    size = ncol * (np.abs(Y[:, rows]) / s[:, None]).max(axis=0)[None, :] * \
        (np.abs(Q) * s[None, :]).max(axis=1)[:, None]
    assert np.all(np.abs(X[:, rows] - ref) <= eps * size)
    ctx.close()


def test_products_over_several_passes(gpu_available):
    """96^3 points of 300 columns take more than one workspace pass; against torch FP64."""
    import torch
    N = (96, 96, 96)
    ncol, Nd = 300, 96 ** 3
    ctx = _ctx(N)
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    Y = torch.rand((ncol, Nd), generator=g, device="cuda", dtype=torch.float64) - 0.5
    HY, X = torch.empty_like(Y), torch.empty_like(Y)
    Hp = torch.empty((ncol, ncol), device="cuda", dtype=torch.float64)
    Mp = torch.empty_like(Hp)
    Q = (torch.rand((ncol, ncol), generator=g, device="cuda", dtype=torch.float64) - 0.5)
    ctx.Project_Hamiltonian(Y, HY, Hp, Mp)
    ctx.Subspace_Rotation(Y, Q, X)
    assert ctx.kernel_status() == 0
    ny, nh = Y.norm(dim=1), HY.norm(dim=1)
    assert ((Mp - Y @ Y.T).abs() / torch.outer(ny, ny)).max() < 1e-12
    assert ((Hp - HY @ Y.T).abs() / torch.outer(nh, ny)).max() < 1e-12
    assert (X - Q @ Y).abs().max() < 1e-12 * ncol * 0.25
    ctx.close()


def test_nonfinite_blocks_follow_the_fp64_gemm(gpu_available):
    """A NaN column and an infinite value: the entries that they touch are not finite, the others
    are those of the clean block."""
    N, ncol = (14, 14, 14), 70
    Nd = 14 ** 3
    rng = np.random.default_rng(2)
    ctx = _ctx(N)
    Y = rng.uniform(-1, 1, (ncol, Nd))
    Q = rng.normal(size=(ncol, ncol))
    Y[5, 100] = np.nan
    Y[9, 200] = np.inf
    HY, Hp, Mp = np.zeros_like(Y), np.zeros((ncol, ncol)), np.zeros((ncol, ncol))
    ctx.Project_Hamiltonian(Y, HY, Hp, Mp)
    ok = [i for i in range(ncol) if i not in (5, 9)]
    assert not np.isfinite(Mp[5]).any() and not np.isfinite(Mp[9, 9])
    ref = Y[ok] @ Y[ok].T
    assert np.abs(Mp[np.ix_(ok, ok)] - ref).max() <= 1e-12 * np.abs(ref).max()
    X = np.zeros_like(Y)
    ctx.Subspace_Rotation(Y, Q, X)
    pts = [i for i in range(Nd) if i not in (100, 200)]
    assert np.isnan(X[:, 100]).all() and not np.isfinite(X[:, 200]).any()
    ref = (Q @ np.nan_to_num(Y, nan=0.0, posinf=0.0))[:, pts]
    assert np.abs(X[:, pts] - ref).max() <= 1e-12 * np.abs(ref).max()
    ctx.close()


def _exact_dot(a, b):
    """The dot product of two FP64 vectors, rounded once: every product split into two exact parts
    (Veltkamp, Dekker), all parts added by math.fsum."""
    import math

    def split(x):
        c = 134217729.0 * x
        hi = c - (c - x)
        return hi, x - hi

    p = a * b
    (ah, al), (bh, bl) = split(a), split(b)
    e = ((ah * bh - p) + ah * bl + al * bh) + al * bl
    return math.fsum(np.concatenate([p, e]))


def test_products_of_a_large_block_are_closer_than_the_fp64_gemm(gpu_available):
    """77^3 points, 520 columns over four decades: Gram entries and rotated values against exact dot
    products. The eight-slice form is off by less than DSYRK and DGEMM are, at worst and on
    average, and by at most 4 units of 2^-53 of the factors' norms."""
    import torch
    N, ncol = (77, 77, 77), 520
    ctx = _ctx(N)
    Nd = 77 ** 3
    g = torch.Generator(device="cuda")
    g.manual_seed(8)
    Y = torch.rand((ncol, Nd), generator=g, device="cuda", dtype=torch.float64) - 0.5
    s = 10.0 ** (4 * torch.rand((ncol, 1), generator=g, device="cuda", dtype=torch.float64) - 2)
    Y *= s
    Q = (torch.rand((ncol, ncol), generator=g, device="cuda", dtype=torch.float64) - 0.5) / s.T
    HY, X = torch.empty_like(Y), torch.empty_like(Y)
    Hp, Mp = torch.empty_like(Q), torch.empty_like(Q)
    rng = np.random.default_rng(9)
    pairs = [(i, i) for i in rng.integers(0, ncol, 6)] + [tuple(p) for p in rng.integers(0, ncol, (14, 2))]
    spots = [(int(n), int(p)) for n, p in zip(rng.integers(0, ncol, 200), rng.integers(0, Nd, 200))]
    err, exact = {}, None
    for mode in (1, 0):
        ctx.set_rr_products(mode)
        ctx.Project_Hamiltonian(Y, HY, Hp, Mp)
        ctx.Subspace_Rotation(Y, Q, X)
        if exact is None:
            y = {i: Y[i].cpu().numpy() for p in pairs for i in p}
            h = {i: HY[i].cpu().numpy() for p in pairs for i in p}
            yp = {p: Y[:, p].cpu().numpy() for _, p in spots}
            q = Q.cpu().numpy()
            exact = ([_exact_dot(y[i], y[j]) for i, j in pairs],
                     [_exact_dot(y[min(p)], h[max(p)]) for p in pairs],
                     [_exact_dot(q[n], yp[p]) for n, p in spots])
            norm = ([np.linalg.norm(y[i]) * np.linalg.norm(y[j]) for i, j in pairs],
                    [np.linalg.norm(y[min(p)]) * np.linalg.norm(h[max(p)]) for p in pairs],
                    [np.linalg.norm(q[n] * s[:, 0].cpu().numpy()) *
                     np.linalg.norm(yp[p] / s[:, 0].cpu().numpy()) for n, p in spots])
        m, hp = Mp.cpu().numpy(), Hp.cpu().numpy()
        # the upper triangle of Yᵀ HY: row the smaller, column the larger index (column-major)
        val = ([m[i, j] for i, j in pairs], [hp[max(p), min(p)] for p in pairs],
               [float(X[n, p]) for n, p in spots])
        err[mode] = [np.abs(np.array(v) - np.array(x)) / np.array(w)
                     for v, x, w in zip(val, exact, norm)]
    ctx.close()
    print("errors (worst, mean) of Mp, Hp, X:",
          {k: [(float(e.max()), float(e.mean())) for e in v] for k, v in err.items()})
    for tc, gemm in zip(err[1], err[0]):
        assert tc.max() <= gemm.max() and tc.mean() <= gemm.mean()
        assert tc.max() <= 4 * 2.0 ** -53
