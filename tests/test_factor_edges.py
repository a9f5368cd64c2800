"""The grid build at its edges: one column, very short and very long series,
singular correlations, designs the fixed point cannot hold, many designs."""

from __future__ import annotations

import copy

import numpy as np
import pytest
import torch

from fastfuncstuff_gb300.glm import grid as G

gpu = pytest.mark.gpu
DEV = torch.device("cuda:0")


def dense_factors(X, a, b, starts, band=None):
    """(logdet R, logdet X'R^-1X, U, G) of one pair in float64, R dense (zero past ``band`` lags where given)."""
    T = X.shape[0]
    a, b = float(np.float32(a)), float(np.float32(b))
    lam = (b + a) * (1 + a * b) / (1 + 2 * a * b + b * b)
    run = np.searchsorted(starts, np.arange(T), side="right")
    gap = np.abs(np.arange(T)[:, None] - np.arange(T)[None, :])
    on = (gap > 0) & (run[:, None] == run[None, :]) & (gap <= (T if band is None else band))
    L = np.linalg.cholesky(np.where(on, lam * a ** np.maximum(gap - 1, 0), 0.0) + np.eye(T))
    Li = np.linalg.inv(L)
    Xw = Li @ X.astype(np.float64)
    C = np.linalg.cholesky(Xw.T @ Xw)
    U = np.linalg.solve(C, Xw.T) @ Li
    return 2 * np.log(np.diag(L) + 1e-10).sum(), 2 * np.log(np.diag(C) + 1e-10).sum(), U, np.linalg.solve(C.T, U)


def check_pair(f, p, pd, X, starts, tol, band=None):
    T = X.shape[0]
    ld_r, ld_x, U, Gm = dense_factors(X, f.grid.a[p], f.grid.b[p], starts, band)
    assert float(f.logdet_R[p]) == pytest.approx(ld_r, rel=1e-9, abs=1e-9)
    assert float(f.logdet_XtX[pd]) == pytest.approx(ld_x, rel=1e-9, abs=1e-9)
    assert np.abs(f.U[pd, :, :T].cpu().numpy() - U).max() <= tol * np.abs(U).max()
    assert np.abs(f.G[pd, :, :T].cpu().numpy() - Gm).max() <= tol * np.abs(Gm).max()


@gpu
@pytest.mark.parametrize("T,banded", [(1100, False), (90, True)])
def test_centring_test_of_one_column_stays_in_its_scratch(T, banded, monkeypatch):
    """K = 1, where the centring test's two vectors are longer than one K x K
    slot: the workspace ends where ffs_grid_work_bytes says (the double past
    it keeps its value), and the pair after (0, 0), whose scratch follows, has
    its dense FP64 factors (a design that is not constant, so a stray
    coefficient would show; fp32 sums of one term: 1e-5)."""
    from fastfuncstuff_gb300.glm import engine

    real = torch.empty

    def filled(*size, **kw):
        t = real(*size, **kw)
        return t.fill_(7.0) if t.dtype == torch.float64 else t

    X = np.random.default_rng(T).standard_normal((T, 1)).astype(np.float32) + 0.5
    Xd = torch.from_numpy(X).to(DEV)
    starts = [0, T // 2]
    G.set_afni_mode(banded, 1e-4)
    try:
        alone = G.make_grid(torch.zeros(1), torch.zeros(1), use_double=True)
        g = G.make_grid(torch.linspace(0.0, 0.6, 3), torch.linspace(-0.4, 0.4, 3), use_double=True)
        monkeypatch.setattr(engine.torch, "empty", filled)
        f1 = engine.build_factors(Xd, alone, G.run_layout(T, starts))
        monkeypatch.undo()
        f = engine.build_factors(Xd, g, G.run_layout(T, starts))
        torch.cuda.synchronize()
    finally:
        G.set_afni_mode(False)
    assert alone.P == 1 and float(f1._keep[3][-1]) == 7.0
    assert int(f1.center_flag) == 0 and int(f.center_flag) == 0
    p = g.p0 + 1
    assert int(f.info.abs().sum()) == 0
    check_pair(f, p, p, X, starts, 1e-5, int(g.band[p]) if banded else None)


@gpu
@pytest.mark.parametrize("T,K,runs,D", [(2, 1, 1, 3), (5, 2, 1, 2), (5, 4, 1, 3), (6, 3, 2, 2), (9, 5, 2, 2), (10, 4, 1, 2)])
def test_many_short_series_against_dense_float64(T, K, runs, D):
    """More items than two waves of series of a few samples, rows padded to a
    multiple of 4 wider than the series. Designs of condition below 30 (fp32
    sums of up to K terms: K 2^-24 30, at least 1e-5)."""
    from fastfuncstuff_gb300.glm import engine

    rng = np.random.default_rng(10 * T + K)
    X = np.stack([np.linalg.qr(rng.standard_normal((T, K)))[0] + 0.05 * d for d in range(D)]).astype(np.float32)
    starts = [T * r // runs for r in range(runs)]
    ax = torch.linspace(-0.8, 0.8, 33)
    g = G.make_grid(ax, ax, use_double=True)
    f = engine.build_factors(torch.from_numpy(X).to(DEV), g, G.run_layout(T, starts), with_tc=True)
    torch.cuda.synchronize()
    assert (f.info.cpu().numpy() == 0).all()
    for d in range(D):
        for p in range(3, g.P, 50):
            check_pair(f, p, d * g.P + p, X[d], starts, max(1e-5, K * 2.0**-24 * 30))


def pivots(a, b, starts, T):
    """(D, m, c) of every sample by the recurrence of D in extended precision; D = 1 where it is not positive."""
    a, b = np.longdouble(np.float32(a)), np.longdouble(np.float32(b))
    lam = (b + a) * (1 + a * b) / (1 + 2 * a * b + b * b)
    D, m, c = np.ones(T, np.longdouble), np.zeros(T, np.longdouble), np.zeros(T, np.longdouble)
    for t in range(T):
        if t not in starts and lam != 0:
            off, c[t] = lam - a, a
            m[t] = off / D[t - 1]
            D[t] = 1 + a * a - 2 * a * lam - m[t] * off
            D[t] = D[t] if D[t] > 0 else 1
    return D, m, c


@gpu
@pytest.mark.parametrize("T,runs,K", [(1024, 1, 4), (1500, 1, 1), (4500, 1, 3), (6400, 1, 1), (6400, 2, 2), (1024, 1, 40)])
def test_long_runs_near_unit_roots(T, runs, K):
    """The LDL' of R where the leading minors leave FP64's range (0.005 a sample
    at (0.99, 0.99)), against the recurrence of D: D to 1e-11 (a rounding of
    the three-term recurrence is amplified by up to 1 / min D), m = off / D
    relative to the largest |m| likewise, then one rounding to fp32."""
    from fastfuncstuff_gb300.glm import engine

    X = np.random.default_rng(T).standard_normal((T, K)).astype(np.float32)
    starts = [T * r // runs for r in range(runs)]
    a, b = np.array([0.0, 0.95, 0.99, 0.99, -0.9, 0.999]), np.array([0.0, 0.95, 0.99, -0.5, -0.9, 0.999])
    ok = (a + b >= 0)
    g = G.grid_of_pairs(a[ok], b[ok], use_double=True)
    f = engine.build_factors(torch.from_numpy(X).to(DEV), g, G.run_layout(T, starts), with_tc=True)
    torch.cuda.synchronize()
    assert int(f.info.abs().sum()) == 0
    coef = f.coef.cpu().numpy().astype(np.float64)
    for p in range(g.P):
        D, m, c = (x.astype(np.float64) for x in pivots(g.a[p], g.b[p], starts, T))
        tol = 1e-11 + 2.0**-24
        for k, want in enumerate((c, m, 1 / D, 1 / np.sqrt(D))):
            assert np.abs(coef[p, :, k] - want).max() <= tol * np.abs(want).max(), (p, k)
        assert float(f.logdet_R[p]) == pytest.approx(2 * np.log(np.sqrt(D) + 1e-10).sum(), rel=1e-11, abs=1e-9)


@gpu
@pytest.mark.parametrize("T,K,D", [(200, 3, 1), (200, 30, 1), (1500, 2, 1), (200, 3, 12)])
def test_singular_correlation_replaces_its_pivots(T, K, D):
    """a = 1: R is all ones, every pivot after a run's first is zero and is
    replaced by 1 (info 2), so logdet R is that of the identity; the other
    pairs have theirs. The item kernel, the wide one and the general one, and
    many designs."""
    from fastfuncstuff_gb300.glm import engine

    X = np.random.default_rng(T).standard_normal((D, T, K)).astype(np.float32)
    starts = [0, T // 2]
    g = copy.deepcopy(G.make_grid(torch.tensor([0.0, 0.5, 0.7]), torch.tensor([0.0, 0.5]), use_double=True))
    g.a[g.a == np.float32(0.7)] = 1.0
    f = engine.build_factors(torch.from_numpy(X if D > 1 else X[0]).to(DEV), g, G.run_layout(T, starts), with_tc=True)
    torch.cuda.synchronize()
    info, coef = f.info.cpu().numpy().reshape(D, g.P), f.coef.cpu().numpy()
    one = g.a == 1.0
    assert one.any() and (info[:, one] == 2).all() and (info[:, ~one] == 0).all()
    for p in range(g.P):
        Dp, m, c = (x.astype(np.float64) for x in pivots(g.a[p], g.b[p], starts, T))
        want = np.stack([c, m, 1 / Dp, 1 / np.sqrt(Dp)], 1)
        assert np.abs(coef[p] - want).max() <= 1e-6 * np.abs(want).max()
        assert float(f.logdet_R[p]) == pytest.approx(2 * np.log(np.sqrt(Dp) + 1e-10).sum(), rel=1e-11, abs=1e-9)


@gpu
@pytest.mark.parametrize("T,K,n", [(400, 24, 3), (600, 130, 3), (1024, 41, 3), (400, 20, 33), (855, 18, 33)])
@pytest.mark.parametrize("kind", ["gaussian", "outlier", "graded", "constant"])
def test_gram_matrix_of_wide_builds_against_exact_sums(T, K, n, kind):
    """X'X at (0, 0), where the whitened design is the design, as the build
    forms it in FP64 (the lower triangle of the slot's factor, which the
    factorisation leaves) against sums in extended precision, whatever the
    columns' profile. Error of an entry over |x_i| |x_j|: a fixed point of
    norm 2^56.4 or more rounds each sample by half a unit (sqrt(T) 2^-56.4 for
    both columns), the products of the low halves left out are at most T 2^52
    of 2^112.8, and the value takes two FP64 roundings."""
    from fastfuncstuff_gb300.glm import engine

    rng = np.random.default_rng(T + K)
    X = rng.standard_normal((T, K))
    if kind == "outlier":
        X[T // 3] *= 1e4
    elif kind == "graded":
        X *= 10.0 ** rng.uniform(-6, 6, (T, K))
    elif kind == "constant":  # every low half alike, no two columns parallel
        X = np.where(np.arange(T)[:, None] % (K + 1) == np.arange(K)[None, :], 2.0, 1.0) * np.linspace(1.0, 1.9, K)
    X = X.astype(np.float32)
    ax = torch.linspace(-0.8, 0.8, n)
    g = G.make_grid(ax, ax, use_double=True)
    f = engine.build_factors(torch.from_numpy(X).to(DEV), g, G.run_layout(T, [0]), with_tc=True)
    torch.cuda.synchronize()
    assert int(f.info[g.p0]) == 0
    slot = 4 * T + 2 * K * T + 4 * K * K
    at = g.p0 * slot + 4 * T + 2 * K * T
    got = f._keep[3][at : at + K * K].cpu().numpy().reshape(K, K)
    Xl = X.astype(np.longdouble)
    want = Xl.T @ Xl
    norm = np.sqrt(np.diag(want))
    err = np.abs(got - want) / (norm[:, None] * norm[None, :])
    tol = np.sqrt(T) * 2.0**-56.4 + T * 2.0**-60.8 + 2.0**-52
    assert (err[np.tril_indices(K)] <= tol).all(), float(err[np.tril_indices(K)].max())


@gpu
@pytest.mark.parametrize("T,K,runs,D,n,zero", [
    (200, 8, 1, 20, None, False),   # one design: the item kernel; all: the wide one, 128 threads
    (331, 13, 2, 9, None, False),
    (300, 20, 3, 7, 21, False),
    (850, 22, 1, 2, 21, False),     # the wide one, 320 threads
    (150, 18, 11, 12, None, False),  # more runs than a warp per run, several runs a time segment
    (97, 1, 1, 30, None, False),
    (120, 7, 2, 20, None, True),    # rank deficient: Gram-Schmidt in every kernel
    (240, 40, 2, 3, 21, True),
    (1100, 6, 2, 3, None, False),   # the general phases
])
def test_a_design_factors_are_its_own_whatever_is_built_beside_it(T, K, runs, D, n, zero):
    """The factors of each design of a build of many equal those of its build
    alone, bit for bit, across the kernels that the number of items selects."""
    from fastfuncstuff_gb300.glm import engine

    rng = np.random.default_rng(T + K)
    X = rng.standard_normal((D, T, K)).astype(np.float32)
    X[:, :, 0] += 3.0
    if zero:
        X[1, :, K // 2] = 0.0
    layout = G.run_layout(T, [T * r // runs for r in range(runs)])
    ax = G.get_default_arma_grids() if n is None else (torch.linspace(-0.8, 0.8, n),) * 2
    g = G.make_grid(*ax)
    kw = dict(task_indices=[0, K // 2], glt=np.eye(K, dtype=np.float32)[:1], with_tc=True, afull=True) if K > 1 else {}
    Xd = torch.from_numpy(X).to(DEV)
    f = engine.build_factors(Xd, g, layout, **kw)
    for d in (0, 1, D - 1):
        one, part = engine.build_factors(Xd[d], g, layout, **kw), engine.design_view(f, d)
        torch.cuda.synchronize()
        assert int(one.info.max()) == (1 if zero and d == 1 else 0)
        for name in ("coef", "logdet_R", "logdet_XtX", "U", "G", "Adiag", "XtX", "info", "Ftask", "glt_var", "uexp",
                     "Afull", "U_hi", "U_lo"):
            a, b = getattr(one, name), getattr(part, name)
            if a is not None:
                assert torch.equal(a.reshape(-1).view(torch.uint8), b.reshape(-1).view(torch.uint8)), (d, name)


@gpu
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("T,K", [(150, 5), (400, 40), (150, 50), (1100, 5)])
def test_design_basis_of_a_design_that_is_not_finite(value, T, K):
    """A sample of the design that is not finite leaves no basis of its column
    (none of it finite) and no centring, whichever way the Gram entries are
    summed (fixed point up to 40 columns and 1,024 samples, else FP64)."""
    from fastfuncstuff_gb300.glm import engine

    X = np.random.default_rng(K).standard_normal((T, K)).astype(np.float32)
    X[:, 0] = 1.0
    X[T // 2, 2] = value
    q0, flag, coef = engine.design_basis(torch.from_numpy(X).to(DEV), with_constant=True)
    torch.cuda.synchronize()
    assert not torch.isfinite(q0[2, :T]).any()
    assert int(flag) == 0 and (coef == 0).all()


@gpu
@pytest.mark.parametrize("T,K,runs,n", [(150, 8, 1, None), (203, 20, 3, 33), (203, 57, 3, None), (400, 130, 2, 3),
                                        (1100, 6, 1, None)])
def test_a_zero_column_goes_through_the_general_phases(T, K, runs, n):
    """A column of zeros has no positive pivot: every kernel of the build sends
    the item to the general phases (info 1), whose basis spans the other
    columns: U'U = L^-T Q Q'L^-1 against a float64 QR of them (sums of K fp32
    products on designs of condition below 30: K 2^-24 30, at least 1e-5)."""
    from fastfuncstuff_gb300.glm import engine

    rng = np.random.default_rng(T + K)
    X = rng.standard_normal((T, K)).astype(np.float32)
    X[:, K // 2] = 0.0
    starts = [T * r // runs for r in range(runs)]
    ax = G.get_default_arma_grids() if n is None else (torch.linspace(-0.8, 0.8, n),) * 2
    g = G.make_grid(*ax, use_double=True)
    f = engine.build_factors(torch.from_numpy(X).to(DEV), g, G.run_layout(T, starts), with_tc=True)
    torch.cuda.synchronize()
    assert (f.info.cpu().numpy() == 1).all()
    rest = np.delete(X, K // 2, 1)
    for p in range(0, g.P, max(1, g.P // 4)):
        _, ld_x, U, _ = dense_factors(rest, g.a[p], g.b[p], starts)
        got = f.U[p, :, :T].cpu().numpy().astype(np.float64)
        assert (got[K // 2] == 0).all()
        want = U.T @ U
        assert np.abs(got.T @ got - want).max() <= max(1e-5, K * 2.0**-24 * 30) * np.abs(want).max()
        # log |R_jj| + 1e-10 of the zero column
        assert float(f.logdet_XtX[p]) == pytest.approx(ld_x + 2 * np.log(1e-10), rel=1e-9)


@gpu
@pytest.mark.parametrize("T,K,runs", [(200, 8, 1), (331, 13, 2), (400, 20, 4), (300, 31, 1), (1100, 12, 2)])
def test_design_basis_is_the_grid_builds_to_rounding(T, K, runs):
    """Q0 and U of (0, 0) come from FP64 factors that agree to their rounding
    (the Gram entries' fixed points differ), rounded to fp32 each and carried
    through the same fp32 recursion: within 4 roundings a column, K 2^-22 of
    the largest entry on designs of condition below 4."""
    from fastfuncstuff_gb300.glm import engine

    X = np.random.default_rng(T).standard_normal((T, K)).astype(np.float32)
    assert np.linalg.cond(X.astype(np.float64)) < 4
    g = G.make_grid(*G.get_default_arma_grids())
    Xd = torch.from_numpy(X).to(DEV)
    f = engine.build_factors(Xd, g, G.run_layout(T, [T * r // runs for r in range(runs)]))
    q0 = engine.design_basis(Xd)
    torch.cuda.synchronize()
    assert float((q0 - f.U[g.p0]).abs().max()) <= K * 2.0**-22 * float(q0.abs().max())


@gpu
@pytest.mark.parametrize("T,K,n", [(200, 8, None), (300, 20, 33), (400, 24, 3), (600, 70, 3)])
@pytest.mark.parametrize("low,high", [(-10, 10), (-17, 17)])
def test_columns_of_any_magnitude(T, K, n, low, high):
    """Columns from 10^low to 10^high: within the fixed point's norms and past
    them (the general phases). The basis does not depend on the columns'
    magnitudes: U against dense float64 (condition below 30 without them)."""
    from fastfuncstuff_gb300.glm import engine

    rng = np.random.default_rng(K)
    mag = 10.0 ** np.linspace(low, high, K)
    X = (rng.standard_normal((T, K)) * rng.permutation(mag)).astype(np.float32)
    ax = G.get_default_arma_grids() if n is None else (torch.linspace(-0.8, 0.8, n),) * 2
    g = G.make_grid(*ax, use_double=True)
    f = engine.build_factors(torch.from_numpy(X).to(DEV), g, G.run_layout(T, [0]), with_tc=True)
    torch.cuda.synchronize()
    assert (f.info.cpu().numpy() == 0).all()
    for p in range(0, g.P, max(1, g.P // 4)):
        scaled = X.astype(np.float64) / np.linalg.norm(X.astype(np.float64), axis=0)
        U = dense_factors(scaled, g.a[p], g.b[p], [0])[2]
        assert np.abs(f.U[p, :, :T].cpu().numpy() - U).max() <= max(1e-5, K * 2.0**-24 * 30) * np.abs(U).max()
