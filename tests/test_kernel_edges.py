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


# ------------------------------------------------------------------ the hierarchical descent


def grid_for(n):
    a, b = G.get_default_arma_grids() if n is None else (torch.linspace(-0.8, 0.8, n),) * 2
    return G.make_grid(a, b)


def full_descent(surf, g):
    """(pair, value) of the selector over a whole surface, read as the reference reads it."""
    n_a, n_b = g.lattice.shape
    value = lambda c: np.inf if g.lattice[c] < 0 else surf[g.lattice[c]]
    cell = (g.za, g.zb)
    low = value(cell)
    for lev in range(g.ltop, -1, -1):
        s = 1 << lev
        if lev == g.ltop:
            cand = [(i, j) for j in range(0, n_b, s) for i in range(0, n_a, s)]
        else:
            cand = [(min(max(cell[0] + i * s, 0), n_a - 1), min(max(cell[1] + j * s, 0), n_b - 1))
                    for j in (-1, 0, 1) for i in (-1, 0, 1)]
        best = cand[0]
        for c in cand[1:]:
            if value(c) < value(best):
                best = c
        if value(best) < low:
            cell, low = best, value(best)
    return int(g.lattice[cell]), low


@pytest.mark.parametrize("n", [None, 5, 9, 17, 18, 21, 33])
@pytest.mark.parametrize("afni", [False, True])
def test_descent_plan_reads_what_the_selector_reads(n, afni):
    """The plan walked on the host over random and smooth surfaces gives the
    whole surface's selection, for lattices of every divisibility (identity
    pairs share one value, as they do in the criterion)."""
    G.set_afni_mode(afni)
    try:
        g = grid_for(n)
    finally:
        G.set_afni_mode(False)
    p = G.descent_plan(g)
    ident = G.lambda_is_zero(g.a, g.b)
    rng = np.random.default_rng(n or 1)
    n_b = g.lattice.shape[1]
    for k in range(60):
        if k % 2:
            surf = rng.standard_normal(g.P)
        else:
            surf = (g.a - rng.uniform(-0.8, 0.8)) ** 2 + (g.b - rng.uniform(-0.8, 0.8)) ** 2 + rng.uniform(-1, 1) * g.a * g.b
        surf[ident] = surf[g.p0]
        seen = np.full(g.P, np.inf)  # only what the first levels evaluate
        seen[p.slots[p.slots >= 0]] = surf[p.slots[p.slots >= 0]]
        seen[ident] = surf[ident]
        on = p.lat_slot.reshape(g.lattice.shape)
        assert all(on[c] == -2 if ident[g.lattice[c]] else p.slots[on[c]] == g.lattice[c] for c in zip(*np.nonzero(on != -1)))
        # the first levels, then one round per level left
        n_a = g.lattice.shape[0]
        val = lambda c: np.inf if on[c] == -1 else seen[g.lattice[c]]
        at = (g.za, g.zb)
        low = val(at)
        for lev in range(g.ltop, p.n_rounds - 1, -1):
            s = 1 << lev
            cand = ([(i, j) for j in range(0, n_b, s) for i in range(0, n_a, s)] if lev == g.ltop else
                    [(min(max(at[0] + i * s, 0), n_a - 1), min(max(at[1] + j * s, 0), n_b - 1))
                     for j in (-1, 0, 1) for i in (-1, 0, 1)])
            best = min(range(len(cand)), key=lambda i: (val(cand[i]), i))
            if val(cand[best]) < low:
                at, low = cand[best], val(cand[best])
        cell = int(g.lattice[at])
        for r in range(p.n_rounds):
            own = p.cell_slots[p.cell_group[r, cell]]
            lst = {int(e) >> 24: int(e) & 0xFFFFFF for e in p.cell_list[r, cell] if e >= 0}
            mn, to = np.inf, -1
            for s in range(8):
                q = int(p.cell_pairs[r, cell, s])
                assert (own[s] == q and lst[s] == q) if q >= 0 else (own[s] == -1 and s not in lst)
                d = surf[q] if q >= 0 else np.inf if q == -1 else surf[-2 - q]
                if d < mn:
                    mn, to = d, q if q >= 0 else -2 - q
            if mn < low:
                low, cell = mn, to
        assert (cell, low) == full_descent(surf, g)


@gpu
@pytest.mark.parametrize("V,T,K,runs,n", [
    (1, 40, 3, 1, None),      # one voxel
    (63, 97, 8, 1, 33),       # a partial tile, T odd
    (257, 200, 9, 2, 33),     # a row past two tiles; a run start inside a block of 16
    (700, 250, 33, 3, 21),    # T % 4 == 2; two blocks of pairs per tile (K > 32)
    (300, 160, 130, 1, 33),   # one pair per block of the projection
    (4096, 128, 20, 1, 18),   # cells clamped at the lattice's edge, whole tiles
    (1500, 72, 6, 4, 41),     # three rounds
])
def test_descent_equals_the_full_surface(V, T, K, runs, n, monkeypatch):
    """best and the criterion there, bit for bit, with zero, constant, huge and NaN series among the voxels."""
    from fastfuncstuff_gb300.glm import engine

    Y, X, starts = arma_data(7, V, T, K, runs, baseline=50.0)
    if V > 60:
        Y[3], Y[17], Y[40], Y[41, 5] = 0.0, 12.5, Y[40] * 1e18, np.nan
    g = grid_for(n)
    Yd, Xd = torch.from_numpy(Y).to(DEV), torch.from_numpy(X).to(DEV)
    f = engine.build_factors(Xd, g, G.run_layout(T, starts))
    monkeypatch.setattr(engine, "DESCENT_MIN_WORK", 0)
    monkeypatch.setattr(engine, "DESCENT_SHARE", 0)
    assert engine._descent_plan(f, V) is not None
    got = engine.search(Yd, f)
    want = engine.search(Yd, f, keep_surface=True)
    assert torch.equal(got.best, want.best)
    assert torch.equal(got.best_crit.view(torch.int32), want.best_crit.view(torch.int32))
    assert torch.equal(got.scale, want.scale) or V > 60


@gpu
@pytest.mark.parametrize("V,T,K,D,n", [(900, 100, 7, 3, 33), (2100, 133, 18, 5, 17), (40, 90, 40, 2, None)])
def test_grouped_descent_equals_the_full_surface(V, T, K, D, n, monkeypatch):
    """One design per group, groups of unequal size (one of them a single voxel), two runs."""
    from fastfuncstuff_gb300.glm import engine

    Y, X, starts = arma_data(9, V, T, K, 2)
    Xs = np.stack([X + 0.1 * d * np.random.default_rng(d).standard_normal(X.shape).astype(np.float32) for d in range(D)])
    gid = np.minimum(np.random.default_rng(2).zipf(1.5, V) - 1, D - 1)
    gid[:] = np.where(gid == D - 1, 0, gid)
    gid[5] = D - 1
    g = grid_for(n)
    Yd, Xd = torch.from_numpy(Y).to(DEV), torch.from_numpy(Xs.astype(np.float32)).to(DEV)
    f = engine.build_factors(Xd, g, G.run_layout(T, starts))
    slots = engine.design_slots(gid, D, K, g.P, DEV)
    monkeypatch.setattr(engine, "DESCENT_SHARE", 0)
    monkeypatch.setattr(engine, "DESCENT_MIN_WORK", 0)
    got = engine.search_designs(Yd, f, slots)
    monkeypatch.setattr(engine, "DESCENT_MIN_WORK", 1 << 60)
    want = engine.search_designs(Yd, f, slots)
    assert torch.equal(got.best, want.best) and torch.equal(got.best_crit, want.best_crit)


# ------------------------------------------------------------------ given (a, b)


@gpu
@pytest.mark.parametrize("V,levels", [(1, 1), (300, 3), (5000, 70), (40000, 40000)])
def test_distinct_pairs_equal_np_unique(V, levels):
    """One voxel, heavy repetition, more pairs than one read-back holds; -0 among them; NaN refused."""
    from fastfuncstuff_gb300.glm import engine

    rng = np.random.default_rng(V)
    ab = rng.uniform(-0.9, 0.9, (levels, 2)).astype(np.float32)[rng.integers(0, levels, V)]
    if V > 1:
        ab[0], ab[V // 2] = (0.0, -0.0), (-0.0, 0.0)
    pairs, index = engine.distinct_pairs(torch.from_numpy(ab), DEV)
    want, inv = np.unique(ab, axis=0, return_inverse=True)
    np.testing.assert_array_equal(pairs, want)
    np.testing.assert_array_equal(index.cpu().numpy(), inv.reshape(-1))
    ab[V - 1, 1] = np.nan
    assert engine.distinct_pairs(torch.from_numpy(ab), DEV) is None


@gpu
@pytest.mark.parametrize("T", [2, 31, 33, 397, 1024])
def test_series_sd_is_the_float_nearest_the_float64_value(T):
    """Compensated sums carry about 48 bits, so the result is within 0.5 ulp
    (+ 2^-20) of the float64 standard deviation, for large baselines, huge and
    tiny values; constant rows and NaN as the float64 expression gives them."""
    from fastfuncstuff_gb300.glm import engine

    rng = np.random.default_rng(T)
    Y = rng.standard_normal((70, T)).astype(np.float32)
    Y[:20] += np.float32(1e4)
    Y[20:30] *= np.float32(1e25)
    Y[30:40] *= np.float32(1e-22)
    Y[40], Y[41], Y[42, 0] = 0.0, 3.7, np.nan
    got = engine.voxel_scale(torch.from_numpy(Y).to(DEV)).cpu().numpy()
    want = Y.astype(np.float64).std(1, ddof=1)
    assert np.isnan(got[42])
    floor = want < 1e-8
    assert (got[floor] == np.float32(1e-8)).all()
    ok = ~floor & ~np.isnan(want)
    ulp = np.spacing(want[ok].astype(np.float32)).astype(np.float64)
    assert (np.abs(got[ok].astype(np.float64) - want[ok]) <= (0.5 + 2.0**-20) * ulp + 1e-15 * want[ok]).all()


# ------------------------------------------------------------------ the proposal network


@gpu
@pytest.mark.parametrize("B", [1, 63, 64, 65, 700, 10300])
def test_mlp_tiles_against_the_oracle(B):
    """Partial, single and several tiles per CTA (64 samples each), with an index list. Sums of B <= 10300 terms
    of one sign pattern: relative error of each gradient below 64-term chains, CTA sums and atomics in float32,
    against the gradient's largest entry: 2^-24 (64 + ceil(B / 64) + 64) <= 2e-5."""
    from fastfuncstuff_gb300.glm import learned
    from oracle import mlp as om

    rng = np.random.default_rng(B)
    p = (om.init(2) + 0.02 * rng.standard_normal(om.N_PARAMS)).astype(np.float32)
    x = rng.standard_normal((B + 5, om.N_IN)).astype(np.float32)
    y = (rng.standard_normal((B + 5, 2)) * 0.4).astype(np.float32)
    idx = rng.permutation(B + 5)[:B].astype(np.int32)
    pt, xt, yt, it = (torch.from_numpy(v).to(DEV) for v in (p, x, y, idx))
    out = learned.ArmaProposal(pt).forward(xt[:B].contiguous()).cpu().numpy()
    np.testing.assert_allclose(out, om.forward(p, x[:B]), rtol=1e-4, atol=1e-5)
    grad, loss = torch.zeros(om.N_PARAMS, device=DEV), torch.zeros(1, device=DEV)
    learned.mlp_grad(pt, xt, yt, it, B, grad, loss)
    L, g = om.loss_and_grad(p.astype(np.float64), x[idx].astype(np.float64), y[idx].astype(np.float64))
    assert np.abs(grad.cpu().numpy() - g).max() <= 2e-5 * np.abs(g).max()
    assert float(loss.item()) == pytest.approx(L, rel=2e-5)


@gpu
@pytest.mark.parametrize("T,K,runs,hole,a_max,corcut", [
    (16, 1, 1, (0, 0), 0.3, 1e-2),      # a history of 16, one column
    (75, 17, 3, (20, 9), 0.8, 1e-4),    # a history of 48, odd runs, censored rows, two rounds of columns
    (130, 5, 1, (60, 50), 0.8, 1e-4),   # one run; a gap wider than the band
    (131, 33, 2, (0, 0), 0.8, 1e-12),   # a history of 128 (band 125), longer than a run
    (40, 4, 4, (0, 0), 0.7, 1e-4),      # runs shorter than the band
])
def test_banded_factors_and_surface_against_dense_float64(T, K, runs, hole, a_max, corcut):
    """AFNI's banded R: its factor, U = L^-T Q and the criterion's y'R^-1 y
    against dense FP64 at the edges of the band's chunks and register
    histories. band_L is FP64 throughout (1e-11 of 1); U leaves as fp32 after
    an fp32 Q and substitution, its error below K fp32 roundings times ||L^-1||
    (1e-5 of the largest entry); a sum of T squares of fp32 recurrences,
    each step within band + 2 roundings that ||L^-1|| carries on, within 3e-5."""
    from fastfuncstuff_gb300.glm import engine

    rng = np.random.default_rng(T + K)
    X = np.concatenate([np.ones((T, 1)), rng.standard_normal((T, K - 1))], 1)
    keep = np.array([t for t in range(T + hole[1]) if not hole[0] <= t < hole[0] + hole[1]])
    starts = [T * r // runs for r in range(runs)]
    G.set_afni_mode(True, corcut)
    try:
        g = G.make_grid(torch.linspace(0.0, a_max, 4), torch.linspace(-0.8, 0.8, 5), use_double=True)
        layout = G.run_layout(T, starts, tau=keep)
        f = engine.build_factors(torch.from_numpy(X.astype(np.float32)).to(DEV), g, layout, with_tc=True)
        V = 300
        Y = torch.from_numpy((rng.standard_normal((V, T)) * 3 + 100).astype(np.float32)).to(DEV)
        out = engine.search(Y, f, keep_surface=True, keep_yr=True)
        torch.cuda.synchronize()
    finally:
        G.set_afni_mode(False)
    assert int(f.info.abs().sum()) == 0
    run_of = np.searchsorted(starts, np.arange(T), side="right")
    gap = np.abs(keep[:, None] - keep[None, :])
    X64 = X.astype(np.float32).astype(np.float64)
    yr = out.yr_t.cpu().numpy().astype(np.float64)
    surf = out.surf.cpu().numpy().astype(np.float64)
    U0 = f.U[g.p0, :, :T].cpu().numpy().astype(np.float64)
    rss0 = (yr ** 2).sum(0) - ((U0 @ yr) ** 2).sum(0)
    base = float(f.logdet_R[g.p0] + f.logdet_XtX[g.p0])
    for p in range(g.P):
        bw = int(g.band[p])
        a, b = float(np.float32(g.a[p])), float(np.float32(g.b[p]))
        lam = (b + a) * (1 + a * b) / (1 + 2 * a * b + b * b)
        R = np.where((gap > 0) & (gap <= bw) & (run_of[:, None] == run_of[None, :]),
                     lam * a ** np.maximum(gap - 1, 0), 0.0) + np.eye(T)
        got = np.zeros((T, T))
        for j in range(f.band_w):
            got[np.arange(j, T), np.arange(T - j)] = f.band_L[p, j:, j].cpu().numpy()
        np.testing.assert_allclose(got, np.linalg.cholesky(R), rtol=0, atol=1e-11, err_msg=f"pair {p}")
        Li = np.linalg.inv(got)
        Xw = Li @ X64
        U = f.U[p, :, :T].cpu().numpy().astype(np.float64)
        want = np.linalg.solve(np.linalg.cholesky(Xw.T @ Xw), Xw.T) @ Li
        assert np.abs(U - want).max() <= 1e-5 * np.abs(want).max()
        ssw, proj = ((Li @ yr) ** 2).sum(0), ((want @ yr) ** 2).sum(0)
        crit = float(f.logdet_R[p] + f.logdet_XtX[p]) - base + (T - K) * np.log1p((ssw - proj - rss0) / rss0)
        scale = (ssw + proj) / np.minimum(ssw - proj, rss0)
        assert (np.abs(surf[p] - crit) <= 3e-5 * (T - K) * scale + 1e-5 * np.abs(crit)).all()


@gpu
@pytest.mark.parametrize("T,K,runs,dup", [
    (161, 41, 1, False),   # the narrowest wide design, four sample slices, T odd
    (203, 57, 3, False),   # runs that start inside a word of four
    (400, 72, 2, False),   # two slices
    (301, 103, 3, False),  # two rounds of blocks
    (600, 130, 1, False),
    (400, 150, 2, False),
    (203, 57, 3, True),    # a repeated column: the general phases' QR
])
def test_wide_designs_against_dense_float64(T, K, runs, dup):
    """Builds of more than 40 columns: Gram matrix, logdets, diag((X'R^-1X)^-1),
    U = L^-T Q and G against dense FP64. The Gram matrix, the factor and its
    inverse are FP64 or finer and leave as fp32 (one rounding, 1e-6 with room
    for the factor's); Q, U and G go through fp32 sums of up to K terms on a
    design of condition below 30 (K 2^-24 30: 3e-4 of the largest entry at
    the widest)."""
    from fastfuncstuff_gb300.glm import engine

    rng = np.random.default_rng(T + K)
    X = rng.standard_normal((T, K)).astype(np.float32)
    X[:, 0] = 1.0
    if dup:
        X[:, 7] = X[:, 3]
    starts = [T * r // runs for r in range(runs)]
    g = G.make_grid(torch.linspace(0.0, 0.8, 3), torch.linspace(-0.4, 0.4, 3), use_double=True)
    f = engine.build_factors(torch.from_numpy(X).to(DEV), g, G.run_layout(T, starts), with_tc=True)
    torch.cuda.synchronize()
    info = f.info.cpu().numpy()
    if dup:
        assert (info == 1).any() or np.isfinite(f.U.cpu().numpy()).all()
        return
    assert (info == 0).all()
    run_of = np.searchsorted(starts, np.arange(T), side="right")
    gap = np.abs(np.arange(T)[:, None] - np.arange(T)[None, :])
    tol = K * 2.0 ** -24 * 30
    for p in range(g.P):
        a, b = float(np.float32(g.a[p])), float(np.float32(g.b[p]))
        lam = (b + a) * (1 + a * b) / (1 + 2 * a * b + b * b)
        R = np.where((gap > 0) & (run_of[:, None] == run_of[None, :]), lam * a ** np.maximum(gap - 1, 0), 0.0) + np.eye(T)
        Li = np.linalg.inv(np.linalg.cholesky(R))
        Xw = Li @ X.astype(np.float64)
        N = Xw.T @ Xw
        C = np.linalg.cholesky(N)
        Ci = np.linalg.inv(C)
        U = (Ci @ Xw.T) @ Li
        np.testing.assert_allclose(float(f.logdet_XtX[p]), 2 * np.log(np.diag(C) + 1e-10).sum(), rtol=1e-9, atol=1e-9)
        np.testing.assert_allclose(f.XtX[p].cpu().numpy(), N, rtol=1e-6, atol=1e-6 * np.abs(N).max())
        np.testing.assert_allclose(f.Adiag[p].cpu().numpy(), np.diag(Ci.T @ Ci), rtol=1e-6)
        got = f.U[p, :, :T].cpu().numpy()
        assert np.abs(got - U).max() <= tol * np.abs(U).max()
        Gm = Ci.T @ U
        assert np.abs(f.G[p, :, :T].cpu().numpy() - Gm).max() <= tol * np.abs(Gm).max()
        assert (f.U[p, :, T:] == 0).all() and (f.G[p, :, T:] == 0).all()
        hi, lo = (x.view(f.P, K, -1)[p].view(torch.float16).double() for x in (f.U_hi, f.U_lo))
        back = ((hi + lo) * 2.0 ** -float(f.uexp[p])).cpu().numpy()[:, :T]
        assert np.abs(back - got).max() <= 2.0 ** -20 * np.abs(got).max()


@gpu
@pytest.mark.parametrize("T", [3, 4, 30, 127, 128, 390, 855])
@pytest.mark.parametrize("V", [1, 33, 300])
def test_prep_scaling_is_the_correctly_rounded_quotient(T, V):
    """(y - m) / s without a design, by corrected products where the values
    are of ordinary size and by divisions elsewhere: the correctly rounded
    quotient, bit for bit, for samples of any magnitude; and the fp16 split of
    it (hi the nearest fp16 of y 2^e, lo of the rest), zero past T."""
    import ctypes as C

    from fastfuncstuff_gb300 import _lib

    rng = np.random.default_rng(T * 1000 + V)
    y = rng.standard_normal((V, T)) * 10.0 ** rng.uniform(-3, 3, (V, 1))
    y[rng.random((V, T)) < 0.05] = 0.0
    y[0, :2] = 1e-25, -3e-22
    if V > 1:
        y[1] = 7.25  # a constant series: the floor of the scale
        y[2 % V] *= 1e18
    Y = torch.from_numpy(y.astype(np.float32)).to(DEV)
    ld = (T + 7) // 8 * 8
    scale = torch.empty(V, device=DEV)
    rows = torch.empty(V, T, device=DEV)
    hi, lo = (torch.full((V, ld), 77, dtype=torch.int16, device=DEV) for _ in range(2))
    yexp = torch.empty(V, dtype=torch.int32, device=DEV)
    a = _lib.PrepArgs(V=V, T=T, K=0, Y=Y.data_ptr(), do_scale=1, center=0, ld_y=ld, scale=scale.data_ptr(),
                      yr_hi=hi.data_ptr(), yr_lo=lo.data_ptr(), yexp=yexp.data_ptr(), yr_rows=rows.data_ptr())
    _lib.check(_lib.load().ffs_reml_prep(C.byref(a), torch.cuda.current_stream().cuda_stream), "ffs_reml_prep")
    torch.cuda.synchronize()
    want = Y.cpu().numpy() / scale.cpu().numpy()[:, None]
    assert np.array_equal(rows.cpu().numpy(), want)
    x = np.ldexp(want.astype(np.float64), yexp.cpu().numpy()[:, None]).astype(np.float32)
    h = x.astype(np.float16)
    low = (x - h.astype(np.float32)).astype(np.float16)
    assert np.array_equal(hi.view(torch.float16).cpu().numpy()[:, :T], h)
    assert np.array_equal(lo.view(torch.float16).cpu().numpy()[:, :T], low)
    assert (hi[:, T:] == 0).all() and (lo[:, T:] == 0).all()


@gpu
@pytest.mark.parametrize("a_max,corcut,lags", [(0.3, 1e-2, 16), (0.8, 1e-4, 48), (0.8, 1e-12, 127)])
def test_banded_gls_whitening_against_dense_float64(a_max, corcut, lags):
    """sigma^2 of the GLS under AFNI's banded R, its tile whitened by 8 lanes a
    row over up to 16, 48 or 127 lags, against the dense FP64 whitening of the
    same fit's residual (fp32 residuals and sums of T squares: 1e-4)."""
    from fastfuncstuff_gb300.glm.arma import fit_glm_arma11

    V, T, K = 70, 131, 4
    Y, X, starts = arma_data(11, V, T, K, runs=2)
    grids = torch.linspace(0.0, a_max, 4), torch.linspace(-0.4, 0.4, 5)
    G.set_afni_mode(True, corcut)
    try:
        g = G.make_grid(*grids)
        r = fit_glm_arma11(torch.from_numpy(Y), torch.from_numpy(X), 2.0, *grids, run_starts=starts, device="cuda",
                           verbose=False)
    finally:
        G.set_afni_mode(False)
    assert lags // 3 < g.band.max() <= lags or lags == 16
    run_of = np.searchsorted(starts, np.arange(T), side="right")
    gap = np.abs(np.arange(T)[:, None] - np.arange(T)[None, :])
    band = {(np.float32(a), np.float32(b)): int(w) for a, b, w in zip(g.a, g.b, g.band)}
    betas, sigma2 = r.betas.numpy().astype(np.float64), r.sigma2.numpy()
    for v in range(V):
        a, b = (np.float32(x) for x in r.arma_params[v].numpy())
        bw, a, b = band[a, b], float(a), float(b)
        lam = (b + a) * (1 + a * b) / (1 + 2 * a * b + b * b)
        R = np.where((gap > 0) & (gap <= bw) & (run_of[:, None] == run_of[None, :]), lam * a ** np.maximum(gap - 1, 0), 0.0)
        w = np.linalg.solve(np.linalg.cholesky(R + np.eye(T)), Y[v] - X.astype(np.float64) @ betas[v])
        assert abs(float(sigma2[v]) - (w @ w) / (T - K)) <= 1e-4 * (w @ w) / (T - K)


@gpu
@pytest.mark.parametrize("T,K,runs,D", [(150, 20, 1, 1), (203, 23, 3, 1), (301, 56, 2, 1), (130, 9, 2, 4), (199, 18, 3, 3)])
def test_many_items_builds_against_dense_float64(T, K, runs, D):
    """Builds of more items than the latency kernel takes (33 x 33 lattice, one
    design or several): logdet, diag((X'R^-1X)^-1), U and G of some pairs
    against dense FP64, to the bounds of the wide designs' test."""
    from fastfuncstuff_gb300.glm import engine

    rng = np.random.default_rng(T + K)
    X = rng.standard_normal((D, T, K)).astype(np.float32)
    X[:, :, 0] = 1.0
    starts = [T * r // runs for r in range(runs)]
    ax = torch.linspace(-0.8, 0.8, 33)
    g = G.make_grid(ax, ax, use_double=True)
    Xd = torch.from_numpy(X if D > 1 else X[0]).to(DEV)
    f = engine.build_factors(Xd, g, G.run_layout(T, starts), with_tc=True)
    torch.cuda.synchronize()
    assert (f.info.cpu().numpy() == 0).all()
    run_of = np.searchsorted(starts, np.arange(T), side="right")
    gap = np.abs(np.arange(T)[:, None] - np.arange(T)[None, :])
    same = (gap > 0) & (run_of[:, None] == run_of[None, :])
    for dsg in range(D):
        for p in range(5, g.P, 90):
            a, b = float(np.float32(g.a[p])), float(np.float32(g.b[p]))
            lam = (b + a) * (1 + a * b) / (1 + 2 * a * b + b * b)
            R = np.where(same, lam * a ** np.maximum(gap - 1, 0), 0.0) + np.eye(T)
            Li = np.linalg.inv(np.linalg.cholesky(R))
            Xw = Li @ X[dsg].astype(np.float64)
            C = np.linalg.cholesky(Xw.T @ Xw)
            Ci = np.linalg.inv(C)
            U = (Ci @ Xw.T) @ Li
            tol = K * 2.0 ** -24 * max(30.0, np.linalg.cond(Xw))
            pd = dsg * g.P + p
            np.testing.assert_allclose(float(f.logdet_XtX[pd]), 2 * np.log(np.diag(C) + 1e-10).sum(), rtol=1e-9, atol=1e-9)
            np.testing.assert_allclose(f.Adiag[pd].cpu().numpy(), np.diag(Ci.T @ Ci), rtol=1e-6)
            assert np.abs(f.U[pd, :, :T].cpu().numpy() - U).max() <= tol * np.abs(U).max()
            Gm = Ci.T @ U
            assert np.abs(f.G[pd, :, :T].cpu().numpy() - Gm).max() <= tol * np.abs(Gm).max()
