"""The performance cases: what a user of this package has it do, through its public entry points.

A case is one call on synthetic fMRI data: V voxels of T retained time points in ``runs`` runs, a design of K columns
(task regressors, a Legendre drift per run, motion random walks), ARMA(1,1) noise with spatially smooth (a, b), every
voxel around a baseline of 100 as percent-signal data are. ``grid`` is 0 for AFNI's default grids (9 x 17 points) or the
n of an n x n grid on [-0.8, 0.8]; 33 is this package's benchmark grid. The kinds:

  fit       fit_glm_arma11, full grid; ``selector`` the default hierarchical descent or the exhaustive argmin,
            ``out`` plain / stats (task columns, GLT contrasts, partial R^2, Ljung-Box), ``io`` device tensors or host arrays
  learned   fit_glm_arma11 with a trained proposal and one re-centred round (``io`` device, or pinned host memory)
  grouped   fit_glm_arma11_grouped: one design per HRF group, censored frames
  refit     fit_glm_arma11 with the (a, b) of an earlier fit (-load_Rvar), residuals and predictions kept
  dsort     fit_glm_arma11 with q voxelwise regressors
  afni      fit_glm_arma11 in AFNI-faithful mode
  surface   search_voxels_precomputed_grid against kept factors, the whole criterion surface returned
  proposal  the proposal network's forward and one gradient of its training (a minibatch)
"""

from __future__ import annotations

import math
import types

import numpy as np
import torch

from fastfuncstuff_gb300 import (
    fit_glm_arma11,
    fit_glm_arma11_grouped,
    get_default_arma_grids,
    precompute_reml_grid,
    search_voxels_precomputed_grid,
    set_afni_mode,
)
from fastfuncstuff_gb300.glm import learned
from fastfuncstuff_gb300.synth import block_drift, double_gamma_hrf, event_regressor

FIELDS = (
    "betas", "tstats", "r2", "sigma2", "fstats", "arma_params", "arma_lambda", "reml_likelihood", "r2_partial",
    "r2_partial_nuisance", "contrast_betas", "contrast_tstats", "contrast_r2_partial", "ljung_box", "residuals",
    "residuals_whitened", "predicted", "dsort_betas", "dsort_tstats",
)


def _case(name, kind, V, T, runs, K, grid, **more):
    c = dict(name=name, kind=kind, V=V, T=T, runs=runs, K=K, grid=grid)
    c.update(more)
    return c


def listed():
    return [
        # one region of interest, host arrays in and out, the default arguments: latency
        _case("roi_host", "fit", 200, 200, 1, 8, 0, selector="hierarchical", out="plain", io="host"),
        # one slice with the statistics a group analysis reads; odd T, odd V
        _case("slice_stats", "fit", 4099, 331, 2, 13, 0, selector="hierarchical", out="stats", io="device"),
        # the whole brain on the benchmark grid, the default selector
        _case("whole_brain", "fit", 200_000, 400, 2, 20, 33, selector="hierarchical", out="plain", io="device"),
        # the same with a trained proposal, data on the device
        _case("learned_brain", "learned", 200_000, 400, 2, 20, 33, io="device"),
        # the same from pinned host memory back to host memory, a smaller mask, T not a multiple of 4
        _case("learned_host", "learned", 100_003, 390, 3, 18, 33, io="host"),
        # HRF groups: 20 designs, four censored runs
        _case("hrf_groups", "grouped", 100_000, 855, 4, 18, 33, groups=20, censored=45),
        # single-trial design, 130 columns
        _case("single_trial", "fit", 30_000, 600, 3, 130, 33, selector="hierarchical", out="plain", io="device"),
        # statistics again at saved (a, b), with the series
        _case("refit_series", "refit", 50_000, 400, 2, 20, 33),
        # two voxelwise regressors (tissue-based nuisance)
        _case("dsort_two", "dsort", 20_000, 300, 2, 16, 0, q=2),
        # AFNI's numbers
        _case("afni_mode", "afni", 6000, 240, 2, 11, 0),
        # likelihood surfaces of a region, factors kept; T odd
        _case("surface_map", "surface", 8000, 397, 2, 20, 33),
        # the proposal network on one training minibatch
        _case("proposal_batch", "proposal", 8192, 0, 0, 0, 0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit", "fit", "fit", "fit", "learned", "learned", "grouped", "grouped", "refit", "dsort", "afni",
                       "surface", "proposal"])
    if kind == "proposal":
        return dict(kind=kind, V=_log(rng, 1000, 65536), T=0, runs=0, K=0, grid=0)
    runs = rng.randint(1, 4)
    T = max(_log(rng, 150, 600), 80 * runs)
    K = max(_log(rng, 6, 32), 2 * runs + 2)
    grid = rng.choice([0, 0, 21, 33])
    c = dict(kind=kind, V=_log(rng, 100, 120_000), T=T, runs=runs, K=K, grid=grid)
    if kind == "fit":
        c.update(selector=rng.choice(["hierarchical", "hierarchical", "exhaustive"]), out=rng.choice(["plain", "stats"]),
                 io=rng.choice(["device", "device", "host"]))
        if rng.random() < 0.15:  # single-trial designs
            c.update(K=rng.randint(60, 130), T=max(T, 300), V=_log(rng, 100, 20_000))
    elif kind == "learned":
        c.update(V=_log(rng, 20_000, 150_000), grid=33, K=min(K, 24), io=rng.choice(["device", "host"]))
    elif kind == "grouped":
        c.update(V=_log(rng, 2000, 60_000), K=min(K, 20), groups=rng.randint(2, 12), censored=T // 20)
    elif kind == "refit":
        c.update(V=_log(rng, 100, 60_000))
    elif kind == "dsort":
        c.update(V=_log(rng, 100, 20_000), T=min(T, 320), K=min(K, 20), q=rng.randint(1, 3), grid=rng.choice([0, 21]))
    elif kind == "afni":
        c.update(V=_log(rng, 100, 8000), T=min(T, 320), K=min(K, 20), grid=0)
    elif kind == "surface":
        c.update(V=_log(rng, 100, 12_000))
    return c


# ------------------------------------------------------------------ inputs


def _grids(case):
    if case["grid"] == 0:
        return get_default_arma_grids()
    g = torch.linspace(-0.8, 0.8, case["grid"])
    return g, g


def _run_lens(T, runs):
    return [T // runs + (1 if r < T % runs else 0) for r in range(runs)]


def _layout(case, rng):
    """(run lengths of all frames, kept frames, run starts and tau of the kept ones)"""
    cens = case.get("censored", 0)
    lens = _run_lens(case["T"] + cens, case["runs"])
    n = sum(lens)
    keep = np.sort(rng.choice(n, case["T"], replace=False)) if cens else np.arange(n)
    start = np.concatenate([[0], np.cumsum(lens)])
    run = np.searchsorted(start, keep, side="right") - 1
    tau = keep - start[run]
    starts = [int(np.nonzero(run == r)[0][0]) for r in range(case["runs"])]
    return lens, keep, starts, tau


def _design(rng, lens, keep, K, hrf):
    """(T, K) float32: task regressors, a drift per run, motion random walks (none in a single-trial design)"""
    n, runs = sum(lens), len(lens)
    deg = 2 if K >= 60 else max(0, min(4, (K - 2) // (2 * runs) - 1))
    drift = block_drift(lens, deg)
    left = K - drift.shape[1]
    if K >= 60:  # one column per trial
        tasks = left - 1
        on = np.linspace(10.0, 2.0 * n - 40.0, tasks) + rng.uniform(-1.0, 1.0, tasks)
        cols = [event_regressor(n, [o], hrf) for o in on]
    else:
        tasks = max(1, min(4, left))
        cols = [event_regressor(n, np.sort(rng.uniform(0.0, 2.0 * n - 30.0, max(6, n // 16))), hrf) for _ in range(tasks)]
    motion = np.cumsum(rng.normal(0.0, 0.05, (n, left - tasks)), axis=0)
    return np.column_stack([*cols, drift, motion])[keep].astype(np.float32)


def _uniform_map(gen, V, lo, hi):
    """A spatially smooth map of V values uniform in [lo, hi]: neighbours alike, every value met"""
    x = torch.randn(1, 1, V + 128, generator=gen, device="cuda")
    x = torch.nn.functional.avg_pool1d(x, 65, 1)[0, 0, :V] + 0.02 * torch.randn(V, generator=gen, device="cuda")
    rank = torch.empty(V, device="cuda", dtype=torch.float32)
    rank[x.argsort()] = (torch.arange(V, device="cuda", dtype=torch.float32) + 0.5) / V
    return lo + (hi - lo) * rank


def _noise(gen, lens, a, b):
    """(V, sum(lens)) ARMA(1,1) noise of unit variance, every run on its own after 50 samples"""
    out = []
    sd = torch.sqrt((1 + 2 * a * b + b * b) / (1 - a * a))
    for n in lens:
        e = torch.randn(n + 50, a.numel(), generator=gen, device="cuda")
        y = e[0].clone()
        for t in range(1, n + 50):
            y = torch.addcmul(torch.addcmul(e[t], b, e[t - 1]), a, y)
            e[t - 1] = y
        out.append(e[49 : n + 49] / sd)
    return torch.cat(out).t().contiguous()


def _inputs(case, seed):
    """Everything that the seed decides, before any of the package's own objects"""
    s = types.SimpleNamespace()
    if case["kind"] == "proposal":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        s.x = torch.randn(case["V"], 9, generator=gen, device="cuda").mul_(0.3)
        s.y = torch.rand(case["V"], 2, generator=gen, device="cuda").mul_(1.6).sub_(0.8)
        s.params = learned.init_params(seed % 1000)
        return s
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    V, K = case["V"], case["K"]
    lens, keep, s.starts, s.tau = _layout(case, rng)
    a, b = _uniform_map(gen, V, 0.1, 0.8), _uniform_map(gen, V, -0.5, 0.3)
    noise = _noise(gen, lens, a, b)[:, torch.from_numpy(keep).cuda()]
    D = case.get("groups", 1)
    s.designs = []
    state = rng.bit_generator.state
    for _ in range(D):  # the same events and motion, another HRF
        h = double_gamma_hrf() if D == 1 else double_gamma_hrf(shape1=4.0 + 3.0 * len(s.designs) / D,
                                                              ratio=0.1 + 0.3 * len(s.designs) / D)
        rng.bit_generator.state = state
        s.designs.append(_design(rng, lens, keep, K, h))
    s.groups = np.minimum(rng.zipf(1.6, V) - 1, D - 1).astype(np.int64)
    s.groups[:D] = np.arange(D)
    beta = torch.randn(V, K, generator=gen, device="cuda")
    sigma = 0.5 + 1.5 * torch.rand(V, 1, generator=gen, device="cuda")
    gid = torch.from_numpy(s.groups).cuda()
    Y = noise.mul_(sigma)
    for d in range(D):
        m = (gid == d).nonzero().reshape(-1)
        Y[m] += beta[m] @ torch.from_numpy(s.designs[d]).cuda().t()
    s.Y = Y.add_(100.0)
    s.tasks = [0, 1]
    s.glt = [np.eye(K, dtype=np.float32)[0], np.eye(K, dtype=np.float32)[0] - np.eye(K, dtype=np.float32)[1]]
    if case["kind"] == "refit":  # the grid point nearest to each voxel's (a, b), as an earlier fit saved them
        pa, pb = _pairs(*_grids(case))
        lat = torch.stack([torch.from_numpy(pa), torch.from_numpy(pb)], 1).cuda()
        near = torch.cat([torch.cdist(torch.stack([a, b], 1)[i : i + 65536], lat).argmin(1) for i in range(0, V, 65536)])
        s.saved = lat[near].cpu()
    if case["kind"] == "dsort":
        base = torch.randn(case["q"], case["T"], generator=gen, device="cuda")
        s.dsort = base[None] + 0.3 * torch.randn(V, case["q"], case["T"], generator=gen, device="cuda")
    return s


_PROPOSALS: dict = {}


def _proposal(case):
    """A proposal for this layout and grid, as a user's program keeps one: trained as learned.train_proposal trains it
    (simulated voxels on a design of this kind, labelled with the argmin of their criterion), here with plain torch and
    from fixed seeds, so that every process has the same one."""
    key = (case["T"], case["runs"], case["K"])
    if key in _PROPOSALS:
        return _PROPOSALS[key]
    rng, gen = np.random.default_rng(11), torch.Generator(device="cuda").manual_seed(11)
    lens, keep, starts, tau = _layout(case, rng)
    X, n = _design(rng, lens, keep, case["K"], double_gamma_hrf()), 65_536
    a, b = _pairs(*_grids(case))
    pair = torch.from_numpy(np.stack([a, b], 1)).cuda()
    pick = torch.randint(0, len(a), (n,), generator=gen, device="cuda")
    q = torch.linalg.qr(torch.from_numpy(X).cuda().double())[0]
    y = _noise(gen, lens, pair[pick, 0], pair[pick, 1]).double()
    y -= (y @ q) @ q.t()
    y /= y.std(1, keepdim=True)
    feats, t0 = torch.full((n, 9), case["T"] / 1000.0, dtype=torch.float64, device="cuda"), 0
    feats[:, :8] = 0
    for m in lens:
        for k in range(8):
            feats[:, k] += (y[:, t0 : t0 + m - k - 1] * y[:, t0 + k + 1 : t0 + m]).sum(1)
        t0 += m
    feats[:, :8] /= (y * y).sum(1, keepdim=True)
    best = _Exact(case, X, starts, tau, a, b).surface(y).argmin(0)
    pair[torch.from_numpy(a + b == 0).cuda()] = 0.0  # R = I along the whole line: its middle
    x, lab = feats.float(), pair[best]
    p, off = learned.init_params(3), np.cumsum([0, 64 * 9, 64, 64 * 64, 64, 2 * 64, 2])
    w = [p[off[i] : off[i + 1]].reshape(shape).clone().requires_grad_()
         for i, shape in enumerate([(64, 9), (64,), (64, 64), (64,), (2, 64), (2,)])]
    steps, opt = 2500, torch.optim.Adam(w, lr=4e-3)
    for i in range(steps):
        opt.param_groups[0]["lr"] = 4e-3 * 0.5 * (1 + math.cos(math.pi * i / steps))
        at = torch.randint(0, n, (4096,), generator=gen, device="cuda")
        loss = ((_mlp(w, x[at]) - lab[at]) ** 2).mean()
        opt.zero_grad()
        loss.backward()
        opt.step()
    _PROPOSALS[key] = learned.ArmaProposal(torch.cat([t.detach().reshape(-1) for t in w]).contiguous())
    return _PROPOSALS[key]


def _mlp(w, x):
    h = torch.nn.functional.gelu(x @ w[0].t() + w[1])
    h = torch.nn.functional.gelu(h @ w[2].t() + w[3])
    return h @ w[4].t() + w[5]


def prepare(case, seed):
    s = _inputs(case, seed)
    kind, host = case["kind"], case.get("io") == "host"
    s.kind = kind
    if kind == "proposal":
        s.net = learned.ArmaProposal(s.params)
        s.grad, s.loss = torch.zeros_like(s.params), torch.zeros(1, device="cuda")
        return s
    ag, bg = _grids(case)
    X = torch.from_numpy(s.designs[0]).cuda()
    s.kw = dict(tr=2.0, a_grid=ag, b_grid=bg, run_starts=s.starts if case["runs"] > 1 else None, device="cuda",
                verbose=False, return_device=not host)
    if case.get("censored"):
        s.kw["tau"] = s.tau
    if kind == "surface":
        s.factors = precompute_reml_grid(X, case["T"], ag, bg, "cuda", run_starts=s.kw["run_starts"])
    if kind == "grouped":
        s.by_group = {h: torch.from_numpy(x).cuda() for h, x in enumerate(s.designs)}
    if kind == "learned":
        s.kw.update(proposal=_proposal(case), proposal_recenter=1)
    if kind == "refit":
        s.kw.update(precomputed_arma_params=s.saved, want_residuals=True, want_predicted=True)
    if kind == "dsort":
        s.kw.update(dsort=s.dsort)
    if kind == "fit":
        s.kw.update(force_exhaustive_search=case["selector"] == "exhaustive")
        if case["out"] == "stats":
            s.kw.update(task_indices=s.tasks, glt_labels=["first", "difference"], glt_matrices=s.glt, want_r2_partial=True,
                        want_ljung_box=True)
    s.X = X
    if host:
        s.Y = s.Y.cpu().pin_memory() if kind == "learned" else s.Y.cpu().numpy()
        s.X = X.cpu() if kind == "learned" else s.designs[0]
    return s


def run(s):
    if s.kind == "proposal":
        out = s.net.forward(s.x)
        s.grad.zero_()
        s.loss.zero_()
        learned.mlp_grad(s.params, s.x, s.y, None, s.x.shape[0], s.grad, s.loss)
        return {"out": out, "grad": s.grad, "loss": s.loss}
    if s.kind == "surface":
        params, crit, surface, _ = search_voxels_precomputed_grid(s.X, s.Y, s.factors, "cuda", return_profile=True)
        return {"params": params, "crit": crit, "surface": surface}
    if s.kind == "grouped":
        r = fit_glm_arma11_grouped(s.Y, s.by_group, s.groups, **s.kw)
    elif s.kind == "afni":
        set_afni_mode(True)
        try:
            r = fit_glm_arma11(s.Y, s.X, **s.kw)
        finally:
            set_afni_mode(False)
    else:
        r = fit_glm_arma11(s.Y, s.X, **s.kw)
    return {f: getattr(r, f) for f in FIELDS if getattr(r, f) is not None}


def _selected_pairs(case, P):
    """Pairs whose criterion the case's selector cannot do without"""
    if case["kind"] == "refit":
        return 0
    if case["kind"] == "surface" or case.get("selector") == "exhaustive":
        return P
    if case["kind"] == "learned":
        return 25
    n = 9 if case["grid"] == 0 else case["grid"]
    return min(P, 9 + 8 * max(0, n.bit_length() - 2))


def work(case):
    V, T, K = case["V"], case["T"], case["K"]
    if case["kind"] == "proposal":
        mac = 9 * 64 + 64 * 64 + 64 * 2
        return {"bytes": 4.0 * V * (9 + 2 + 2) + 8.0 * 4994, "flops": 2.0 * V * mac * 4}
    P, D = len(_pairs(*_grids(case))[0]), case.get("groups", 1)
    n_out = V * (2 * K + 6) + (V * P if case["kind"] == "surface" else 0) + (3 * V * T if case["kind"] == "refit" else 0)
    q = case.get("q", 0)
    pairs = _selected_pairs(case, P)
    # residualisation (4KT), each criterion (2KT + 4T), the GLS (6KT), the factors of every pair and design (2TK^2)
    flops = V * (4.0 * K * T + pairs * (2.0 * K * T + 4.0 * T) + 6.0 * K * T + 8.0 * q * K * T) + D * P * 2.0 * T * K * K
    return {"bytes": 4.0 * (V * T * (1 + q) + D * T * K + n_out), "flops": flops}


# ------------------------------------------------------------------ 64 bits


def _pairs(ag, bg):
    """The valid (a, b) in list order, float32: lambda >= 0, decided in float32"""
    ax = []
    for g in (ag, bg):
        g = torch.as_tensor(g, dtype=torch.float32).cpu().clone()
        g[g.abs() < 1e-6] = 0.0
        ax.append(g)
    a, b = (m.reshape(-1) for m in torch.meshgrid(*ax, indexing="ij"))
    ok = (a + b) * (1 + a * b) / (1 + b**2 + 2 * a * b) >= 0
    return a[ok].numpy(), b[ok].numpy()


class _Exact:
    """The ARMA(1,1) REML fit of one design in float64: plain torch, dense in the design, the whitening of the exact R
    through its AR filter (R filtered is tridiagonal) and AFNI's banded R through dense Cholesky factors."""

    def __init__(self, case, X, starts, tau, a, b, band=None):
        self.T, self.K = X.shape
        self.X = torch.from_numpy(X).double().cuda()
        self.a, self.b, self.P = a.astype(np.float64), b.astype(np.float64), len(a)
        self.lam = (self.a + self.b) * (1 + self.a * self.b) / (1 + 2 * self.a * self.b + self.b**2)
        self.dense = band is not None
        bounds = list(zip(starts, [*starts[1:], self.T]))
        if self.dense:
            self._dense(bounds, tau, band)
        else:
            self._filter(bounds, tau)
        XW = self._whiten_design()                                # (P, T, K)
        self.XtX = XW.transpose(1, 2) @ XW
        Lx = torch.linalg.cholesky(self.XtX)
        self.A = torch.cholesky_inverse(Lx)
        self.B = self._unwhiten(XW)                               # R^-1 X
        self.U = torch.linalg.solve_triangular(Lx, self.B.transpose(1, 2), upper=False)  # (P, K, T)
        self.const = self.logdet + 2 * torch.log(torch.diagonal(Lx, dim1=1, dim2=2) + 1e-10).sum(1)

    def _filter(self, bounds, tau):
        c, m, D = np.zeros((self.T, self.P)), np.zeros((self.T, self.P)), np.ones((self.T, self.P))
        on = self.a + self.b != 0
        for t0, t1 in bounds:
            for t in range(t0 + 1, t1):
                g = int(tau[t] - tau[t - 1])
                rho, ct = self.lam * self.a ** (g - 1), self.a**g
                off = rho - ct
                mt = off / D[t - 1]
                c[t], m[t] = np.where(on, ct, 0), np.where(on, mt, 0)
                D[t] = np.where(on, 1 + ct * ct - 2 * ct * rho - mt * off, 1)
        self.c, self.m, self.D = (torch.from_numpy(x).cuda() for x in (c, m, D))
        self.logdet = 2 * torch.log(self.D.sqrt() + 1e-10).sum(0)

    def _dense(self, bounds, tau, band):
        R = np.zeros((self.P, self.T, self.T))
        for t0, t1 in bounds:
            g = np.abs(tau[t0:t1, None] - tau[None, t0:t1])[None]
            r = self.lam[:, None, None] * self.a[:, None, None] ** np.maximum(g - 1, 0)
            R[:, t0:t1, t0:t1] = np.where(g == 0, 1.0, np.where(g <= band[:, None, None], r, 0.0))
        L = torch.linalg.cholesky(torch.from_numpy(R).cuda())
        self.Li = torch.linalg.solve_triangular(L, torch.eye(self.T, dtype=torch.float64, device="cuda").expand_as(L), upper=False)
        self.logdet = 2 * torch.log(torch.diagonal(L, dim1=1, dim2=2) + 1e-10).sum(1)

    def _whiten_design(self):
        if self.dense:
            return self.Li @ self.X
        out = torch.empty(self.P, self.T, self.K, dtype=torch.float64, device="cuda")
        v, xp = torch.zeros(self.P, self.K, dtype=torch.float64, device="cuda"), torch.zeros_like(self.X[0])
        for t in range(self.T):
            v = (self.X[t] - self.c[t, :, None] * xp) - self.m[t, :, None] * v
            out[:, t], xp = v / self.D[t, :, None].sqrt(), self.X[t]
        return out

    def _unwhiten(self, W):
        if self.dense:
            return self.Li.transpose(1, 2) @ W
        out, v = torch.empty_like(W), torch.zeros(self.P, self.K, dtype=torch.float64, device="cuda")
        for t in range(self.T - 1, -1, -1):
            m1, c1 = (self.m[t + 1, :, None], self.c[t + 1, :, None]) if t + 1 < self.T else (0.0, 0.0)
            nv = W[:, t] / self.D[t, :, None].sqrt() - m1 * v
            out[:, t] = nv - c1 * v
            v = nv
        return out

    def surface(self, Y):
        """(P, V) criterion of the series Y (V, T)"""
        Yt = Y.t().contiguous()
        V = Y.shape[0]
        surf = torch.empty(self.P, V, dtype=torch.float64, device="cuda")
        step = max(1, min(self.P, int(1.5e8 // (V * max(self.K, 1))), int(1.2e7 // V)))
        for p in range(0, self.P, step):
            q = min(self.P, p + step)
            if self.dense:
                ss = ((self.Li[p:q] @ Yt) ** 2).sum(1)
            else:
                ss = torch.zeros(q - p, V, dtype=torch.float64, device="cuda")
                v, yp = torch.zeros_like(ss), torch.zeros_like(Yt[0])
                for t in range(self.T):
                    c, m, D = (x[t, p:q, None] for x in (self.c, self.m, self.D))
                    v = torch.addcmul(Yt[t] - c * yp, m, v, value=-1)
                    ss, yp = torch.addcmul(ss, v, v / D), Yt[t]
            proj = (self.U[p:q].reshape(-1, self.T) @ Yt).square_().view(q - p, self.K, V).sum(1)
            rss = (ss - proj).clamp_(min=0)
            surf[p:q] = self.const[p:q, None] + (self.T - self.K) * torch.log(rss + 1e-10)
        return surf

    def whiten(self, R, best):
        """L^-1 of each row of R (V, T) at its own pair"""
        if self.dense:
            out = torch.empty_like(R)
            for p in best.unique().tolist():
                i = (best == p).nonzero().reshape(-1)
                out[i] = R[i] @ self.Li[p].t()
            return out
        Rt = R.t().contiguous()
        out, v, yp = torch.empty_like(Rt), torch.zeros_like(Rt[0]), torch.zeros_like(Rt[0])
        for t in range(self.T):
            v = (Rt[t] - self.c[t][best] * yp) - self.m[t][best] * v
            out[t], yp = v / self.D[t][best].sqrt(), Rt[t]
        return out.t().contiguous()

    def fit(self, Y, scale, best, case, s, D=None):
        """The GLS of every series at its pair, with all the statistics the case asks for"""
        K, T, V = self.K, self.T, Y.shape[0]
        y = Y / scale[:, None]
        rhs = torch.empty(V, K, dtype=torch.float64, device="cuda")
        for p in best.unique().tolist():
            i = (best == p).nonzero().reshape(-1)
            rhs[i] = y[i] @ self.B[p]
        out, q = {}, 0
        if D is None:
            beta = torch.einsum("vij,vj->vi", self.A[best], rhs)
            res, cov = y - beta @ self.X.t(), None
        else:
            q = D.shape[1]
            N = torch.zeros(V, K + q, K + q, dtype=torch.float64, device="cuda")
            N[:, :K, :K] = self.XtX[best]
            for p in best.unique().tolist():
                i = (best == p).nonzero().reshape(-1)
                N[i, :K, K:] = (D[i] @ self.B[p]).transpose(1, 2)
            Dw = torch.stack([self.whiten(D[:, k], best) for k in range(q)], 1)
            N[:, K:, :K] = N[:, :K, K:].transpose(1, 2)
            N[:, K:, K:] = Dw @ Dw.transpose(1, 2) + 1e-8 * torch.eye(q, dtype=torch.float64, device="cuda")
            full = torch.cat([rhs, torch.einsum("vqt,vt->vq", Dw, self.whiten(y, best))], 1)
            cov = torch.linalg.inv(N)
            both = torch.einsum("vij,vj->vi", cov, full)
            beta, bd = both[:, :K], both[:, K:]
            res = y - beta @ self.X.t() - torch.einsum("vq,vqt->vt", bd, D)
        dof = max(1, T - K - q)
        rw = self.whiten(res, best)
        s2 = rw.square().sum(1) / dof
        A = self.A[best] if cov is None else cov[:, :K, :K]
        tstat = beta / ((s2[:, None] * torch.diagonal(A, dim1=1, dim2=2)).sqrt() + 1e-10)
        stats = case.get("out") == "stats"
        if stats:
            ix = torch.tensor(s.tasks, device="cuda")
            M = torch.linalg.inv(A[:, ix][:, :, ix] + 1e-8 * torch.eye(len(ix), dtype=torch.float64, device="cuda"))
            bt = beta[:, ix]
        else:
            M, bt = (self.XtX[best] if cov is None else torch.linalg.inv(A)), beta
        out["fstats"] = torch.einsum("vi,vij,vj->v", bt, M, bt) / (s2 * bt.shape[1] + 1e-10)
        sst = (y - y.mean(1, keepdim=True)).square().sum(1)
        out["r2"] = 1 - res.square().sum(1) / sst
        out["sigma2"] = s2 * scale**2
        unit = scale[:, None]
        out["betas"], out["tstats"] = (beta * unit)[:, s.tasks] if stats else beta * unit, tstat[:, s.tasks] if stats else tstat
        ab = torch.from_numpy(np.stack([self.a, self.b], 1)).cuda()[best]
        out["arma_params"] = ab
        av, bv = ab[:, 0], ab[:, 1]
        out["arma_lambda"] = (av + bv) * (1 + av * bv) / (1 + 2 * av * bv + bv * bv + 1e-10)
        if q:
            out["dsort_betas"] = bd * unit
            out["dsort_tstats"] = bd / ((s2[:, None] * torch.diagonal(cov, dim1=1, dim2=2)[:, K:]).sqrt() + 1e-10)
        if case["kind"] == "refit":
            out["residuals"], out["residuals_whitened"] = res * unit, rw * unit
            out["predicted"] = (y - res) * unit
        if stats:
            part = tstat**2 / (tstat**2 + dof)
            out["r2_partial"] = part[:, s.tasks]
            out["r2_partial_nuisance"] = part[:, [j for j in range(K) if j not in s.tasks]]
            C = torch.from_numpy(np.stack(s.glt)).double().cuda()
            cb = beta @ C.t()
            ct = cb / ((s2[:, None] * torch.einsum("ci,vij,cj->vc", C, A, C)).clamp(min=0).sqrt() + 1e-10)
            out["contrast_betas"], out["contrast_tstats"] = cb * unit, ct
            out["contrast_r2_partial"] = ct**2 / (ct**2 + dof)
            out["ljung_box"] = self._ljung_box(rw, s)
        return out

    def _ljung_box(self, w, s):
        T, K = self.T, self.K
        lens = np.diff([*s.starts, T])
        low = int(lens.min())
        h = min(K + 2 + min(low // 8, int(round(3.0 * math.log(low)))), low // 2)
        if h < 2 or h > T // 2:
            h = min(2 + min(T // 8, int(round(3.0 * math.log(T)))), T // 2)
        total = torch.zeros(w.shape[0], dtype=torch.float64, device="cuda")
        ss = w.square().sum(1)
        for k in range(1, h + 1):
            acc, n = torch.zeros_like(total), 0
            for t0, m in zip(s.starts, lens):
                if m > k:
                    acc += (w[:, t0 : t0 + m - k] * w[:, t0 + k : t0 + m]).sum(1)
                    n += int(m) - k
            if n > 1:
                total += (acc / ss) ** 2 / n
        return (T * (T + 2.0) * total).clamp(max=1e10)


def _hierarchical(surf, a, b, afni):
    """The power-of-two descent from (0, 0) on the lattice of the pairs, per voxel"""
    ax, bx = np.unique(a), np.unique(b)
    lat = np.full((len(ax), len(bx)), -1, np.int64)
    lat[np.searchsorted(ax, a), np.searchsorted(bx, b)] = np.arange(len(a))
    lat = torch.from_numpy(lat).cuda()
    na, nb, V = len(ax), len(bx), surf.shape[1]
    pad = torch.cat([surf, torch.full((1, V), math.inf, dtype=torch.float64, device="cuda")])
    at = torch.arange(V, device="cuda")
    if afni:
        top = max(0, min((na - 1).bit_length() - 1, (nb - 1).bit_length() - 1) - 2)
    else:
        top = max(0, min(na, nb).bit_length() - 2)
    ia = torch.full((V,), int(np.nonzero(np.abs(ax) < 1e-6)[0][0]), device="cuda")
    ib = torch.full((V,), int(np.nonzero(np.abs(bx) < 1e-6)[0][0]), device="cuda")
    low = pad[lat[ia, ib], at]
    for lev in range(top, -1, -1):
        step = 1 << lev
        if lev == top:
            cand = [(torch.full_like(ia, i), torch.full_like(ib, j)) for j in range(0, nb, step) for i in range(0, na, step)]
        else:
            cand = [((ia + i * step).clamp(0, na - 1), (ib + j * step).clamp(0, nb - 1)) for j in (-1, 0, 1) for i in (-1, 0, 1)]
        for i, j in cand:  # the first of equals
            val = pad[lat[i, j], at]
            hit = val < low
            ia, ib, low = torch.where(hit, i, ia), torch.where(hit, j, ib), torch.where(hit, val, low)
    return lat[ia, ib]


def _afni_band(a, b, cor=1e-4):
    """(pairs kept, band of each): AFNI cuts R where lambda rho^(k-1) has fallen to cor"""
    a32, b32 = torch.from_numpy(a), torch.from_numpy(b)
    lam = ((a32 + b32) * (1 + a32 * b32) / (1 + b32**2 + 2 * a32 * b32)).numpy().astype(np.float64)
    ok = (lam == 0) | (lam.astype(np.float32) >= np.float32(cor))
    band = []
    for x, m in zip(a[ok].astype(np.float64), np.abs(lam[ok])):
        rho = max(-0.9, min(0.9, x))
        band.append(0 if m < cor else 1 if rho == 0 else 1 + int(math.ceil(math.log(cor / m) / math.log(abs(rho)))))
    return ok, np.array(band)


def exact(case, seed):
    s = _inputs(case, seed)
    if case["kind"] == "proposal":
        p = s.params.double()
        off = np.cumsum([0, 64 * 9, 64, 64 * 64, 64, 2 * 64, 2])
        w = [p[off[i] : off[i + 1]].reshape(shape).clone().requires_grad_()
             for i, shape in enumerate([(64, 9), (64,), (64, 64), (64,), (2, 64), (2,)])]
        out = _mlp(w, s.x.double())
        loss = ((out - s.y.double()) ** 2).sum() / (2 * s.x.shape[0])
        loss.backward()
        return {"out": out.detach(), "grad": torch.cat([x.grad.reshape(-1) for x in w]), "loss": loss.detach().reshape(1)}
    V, afni = case["V"], case["kind"] == "afni"
    a, b = _pairs(*_grids(case))
    band = None
    if afni:
        ok, band = _afni_band(a, b)
        a, b = a[ok], b[ok]
    Y = s.Y.double()
    scale = Y.std(1)
    D = s.dsort.double() if case["kind"] == "dsort" else None
    gid, outs = torch.from_numpy(s.groups).cuda(), {}
    ident = torch.from_numpy(a + b == 0).cuda()
    first = int(np.nonzero(a + b == 0)[0][0])
    for d, X in enumerate(s.designs):
        i = (gid == d).nonzero().reshape(-1) if len(s.designs) > 1 else torch.arange(V, device="cuda")
        e = _Exact(case, X, s.starts, s.tau, a, b, band)
        if case["kind"] == "refit":
            index = {ab: k for k, ab in enumerate(zip(a.tolist(), b.tolist()))}
            best, crit = torch.tensor([index[tuple(ab)] for ab in s.saved.tolist()], device="cuda"), None
        else:
            parts = []
            for j in range(0, i.numel(), 50_000):
                k = i[j : j + 50_000]
                surf = e.surface(Y[k] / scale[k, None])
                surf[ident] = surf[first].clone()  # one criterion, R = I; the first of them stands for the line
                if case["kind"] in ("learned", "surface") or case.get("selector") == "exhaustive":
                    pick = surf.argmin(0)
                    pick = torch.where(ident[pick], first, pick)
                else:
                    pick = _hierarchical(surf, a, b, afni)
                parts.append((pick, surf.gather(0, pick[None])[0], surf.t() if case["kind"] == "surface" else None))
            best, crit = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])
            if case["kind"] == "surface":
                ab = torch.from_numpy(np.stack([a, b], 1).astype(np.float64)).cuda()
                return {"params": ab[best], "crit": crit, "surface": torch.cat([p[2] for p in parts])}
        got = e.fit(Y[i], scale[i], best, case, s, D)
        got["reml_likelihood"] = crit if crit is not None else torch.zeros(V, dtype=torch.float64, device="cuda")
        for f, v in got.items():
            outs.setdefault(f, torch.empty((V, *v.shape[1:]), dtype=torch.float64, device="cuda"))[i] = v
    return outs
