"""The grid build at its edges: one column, very short and very long series,
singular correlations, designs the fixed point cannot hold, many designs."""

from __future__ import annotations

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
