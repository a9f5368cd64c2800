"""Kernels and dispatch branches at the sizes where they can go wrong: edges
of tiles and words, remainders, the smallest and the largest of a range."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from fastfuncstuff_gb300.glm import grid as G

gpu = pytest.mark.gpu
DEV = torch.device("cuda:0")


def arma_data(seed: int, V: int, T: int, K: int, runs: int = 1, baseline: float = 0.0):
    """(Y (V, T), X (T, K), run starts): seeded ARMA(1,1) voxels on a smooth design with a constant per run."""
    rng = np.random.default_rng(seed)
    starts = [T * r // runs for r in range(runs)]
    ends = [*starts[1:], T]
    X = np.zeros((T, K))
    for r, (s, e) in enumerate(zip(starts, ends)):
        X[s:e, r] = 1.0
    t = np.linspace(-1.0, 1.0, T)
    for j in range(runs, K):
        X[:, j] = np.cos((0.7 + 1.3 * (j - runs)) * np.pi * t + j) + 0.2 * rng.standard_normal(T)
    a, b = rng.uniform(0.1, 0.8, V), rng.uniform(-0.5, 0.3, V)
    Y = np.empty((V, T))
    for s, e in zip(starts, ends):
        ep = rng.standard_normal(V)
        y = ep.copy()
        for i in range(s - 30, e):
            en = rng.standard_normal(V)
            y = a * y + en + b * ep
            ep = en
            if i >= s:
                Y[:, i] = y
    Y += rng.standard_normal((V, K)) @ X.T + baseline
    return Y.astype(np.float32), X.astype(np.float32), starts


# ------------------------------------------------------------------ Ljung-Box


def ljung_box_f64(w, plan):
    """(statistic, T (T + 2) sum |c_k| / n_k) of the rows w by direct binning in float64."""
    h, tau, wt, _ = plan
    T = w.shape[1]
    tau = np.arange(T) if tau is None else tau
    w = w.astype(np.float64)
    bins = np.zeros((w.shape[0], h + 1))
    for k in range(1, h + 1):
        d = tau[k:] - tau[: T - k]
        for t in np.nonzero((d > 0) & (d <= h))[0]:
            bins[:, d[t]] += w[:, t] * w[:, t + k]
    c = bins / (w**2).sum(1, keepdims=True)
    return T * (T + 2.0) * (c**2 * wt).sum(1), T * (T + 2.0) * (np.abs(c) * wt).sum(1)


@gpu
@pytest.mark.parametrize("T,K,runs,censor", [
    (33, 3, 1, 0),     # fewer than 32 lags, one row of lanes and one sample
    (331, 13, 2, 0),   # odd T, two runs
    (400, 20, 2, 0),   # 38 lags: a second 32-lag word
    (400, 60, 1, 0),   # 78 lags: three words
    (361, 18, 4, 39),  # censoring gaps: lags with missing partners
])
def test_ljung_box_lags_against_direct_binning(T, K, runs, censor):
    """The statistic of the returned whitened residuals. Each c_k is a float32
    sum of T products in chains of ceil(T / 32) terms and a 5-step tree, of
    rows rounded once more on output: |error| <= (ceil(T / 32) + 12) 2^-24, as
    sum |w_t w_t+k| <= sum w^2; LB is quadratic in c_k, and its weights and
    result are rounded to float32."""
    from fastfuncstuff_gb300 import fit_glm_arma11

    V = 37
    Y, X, starts = arma_data(3, V, T + censor, K, runs)
    tau, rs = None, starts if runs > 1 else None
    if censor:
        keep = np.sort(np.random.default_rng(5).choice(T + censor, T, replace=False))
        rs, tau = G.build_censor_run_info(starts, T + censor, keep.tolist())
        Y, X = np.ascontiguousarray(Y[:, keep]), np.ascontiguousarray(X[keep])
    got = fit_glm_arma11(Y, X, tr=2.0, device=DEV, verbose=False, run_starts=rs, tau=tau, want_ljung_box=True,
                         want_residuals=True)
    plan = G.ljung_box_plan(T, K, rs, tau)
    want, slope = ljung_box_f64(got.residuals_whitened.numpy(), plan)
    e = (-(-T // 32) + 12) * 2.0**-24
    tol = 2 * e * slope + e * e * T * (T + 2.0) * plan[2].sum() + 4e-7 * want
    assert (np.abs(got.ljung_box.numpy() - want) <= tol).all()
