"""Fits at their edges: long series, groupings that come back, waits that run out."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from fastfuncstuff_gb300.glm import grid as G
from tests.test_kernel_edges import arma_data, ljung_box_f64

gpu = pytest.mark.gpu
DEV = torch.device("cuda:0")


@gpu
@pytest.mark.parametrize("T,K,runs", [(1400, 20, 1), (1400, 20, 2)])
def test_ljung_box_without_room_for_its_table(T, K, runs):
    """A tile of series that leaves no shared memory for the lags' pair table:
    plain index lags summed by shuffles, run-aware ones by atomics. Each c_k is
    a float32 sum of T products: in chains of ceil(T / 32) terms and a 5-step
    tree, |error| <= (ceil(T / 32) + 12) 2^-24 of ssw with the rounding of the
    returned rows, or in one chain of atomics, (T + 12) 2^-24."""
    from fastfuncstuff_gb300 import fit_glm_arma11

    Y, X, starts = arma_data(3, 9, T, K, runs)
    rs = starts if runs > 1 else None
    got = fit_glm_arma11(Y, X, tr=2.0, device=DEV, verbose=False, run_starts=rs, want_ljung_box=True, want_residuals=True)
    plan = G.ljung_box_plan(T, K, rs, None)
    assert (plan[1] is None) == (runs == 1)
    want, slope = ljung_box_f64(got.residuals_whitened.numpy(), plan)
    e = ((-(-T // 32) if runs == 1 else T) + 12) * 2.0**-24
    tol = 2 * e * slope + e * e * T * (T + 2.0) * plan[2].sum() + 4e-7 * want
    assert (np.abs(got.ljung_box.numpy() - want) <= tol).all()


@pytest.mark.parametrize("order,captured", [("AA", "A"), ("AAA", "A"), ("ABAB", "AB"), ("ABBA", "BA"), ("ABCABC", ""),
                                            ("AABABA", "AB"), ("ABCCAB", "C")])
def test_grouped_graphs_are_captured_for_groupings_that_come_back(order, captured, monkeypatch):
    """Captured at the second of two in a row or of two that alternate; three
    in turn, of which the cache would evict each before it returns, never."""
    from fastfuncstuff_gb300.glm import engine

    built = []

    class Plan:
        def __init__(self, Y, Xs, grid, layout, slots, **kw):
            built.append(chr(ord("A") + int(slots.design[0])))

    monkeypatch.setattr(engine, "GroupedFitGraph", Plan)
    monkeypatch.setattr(engine, "_GROUPED_GRAPHS", {})
    monkeypatch.setattr(engine, "_GROUPED_RECENT", {})
    Y, Xs = torch.zeros(6, 20), torch.zeros(3, 20, 2)
    g, layout = G.make_grid(*G.get_default_arma_grids()), G.run_layout(20)
    for name in order:
        gid = np.full(6, ord(name) - ord("A"))
        engine.grouped_graph_for(Y, Xs, g, layout, gid, hierarchical=True, do_scale=True, gls_kw={}, factor_kw={})
    assert "".join(built) == captured


@gpu
def test_grouped_graph_replays_other_data_and_other_designs(monkeypatch):
    """A captured grouped fit replayed on other data, on designs whose span
    lost the constant (the centring flag computed inside the graph goes to 0)
    and on the first ones again equals the eager fit bit for bit; so does one
    of two groupings that alternate."""
    from fastfuncstuff_gb300 import fit_glm_arma11_grouped, synth
    from fastfuncstuff_gb300.glm import engine

    w = synth.workload(2, V=5000)
    keep = np.isin(w.groups, np.arange(4))
    Y, gid = w.Y[keep], w.groups[keep]
    designs = {h: w.designs[h] for h in range(4)}
    assert all(engine.constant_in_span(x) for x in designs.values())
    ramp = dict(designs)
    ramp[2] = designs[2] * (1.0 + np.linspace(0.0, 0.5, Y.shape[1], dtype=np.float32)[:, None])
    assert not engine.constant_in_span(ramp[2])
    other = np.roll(gid, 7)
    kw = dict(a_grid=np.linspace(-0.8, 0.8, 33), b_grid=np.linspace(-0.8, 0.8, 33), run_starts=w.run_starts, tau=w.tau,
              device=DEV, verbose=False, want_residuals=True)
    monkeypatch.setattr(engine, "_GROUPED_GRAPHS", {})
    monkeypatch.setattr(engine, "_GROUPED_RECENT", {})
    monkeypatch.setattr(engine, "DESCENT_MIN_WORK", 0)
    runs, real = [], engine.GroupedFitGraph.run
    monkeypatch.setattr(engine.GroupedFitGraph, "run", lambda self, *a: (runs.append(self), real(self, *a))[1])
    steps = [(Y, designs, gid, 0), (Y, designs, gid, 1), (Y[:, ::-1].copy(), designs, gid, 2), (Y, ramp, gid, 3),
             (Y, designs, gid, 4), (Y, designs, other, 4), (Y, designs, gid, 5), (Y, ramp, other, 6), (Y, ramp, gid, 7)]
    for data, xs, groups, replays in steps:
        graph = fit_glm_arma11_grouped(data, xs, groups, tr=2.0, cuda_graphs=True, **kw)
        assert len(runs) == replays
        eager = fit_glm_arma11_grouped(data, xs, groups, tr=2.0, cuda_graphs=False, **kw)
        for name in ("arma_params", "reml_likelihood", "betas", "tstats", "sigma2", "fstats", "r2", "residuals",
                     "residuals_whitened"):
            np.testing.assert_array_equal(getattr(graph, name).numpy(), getattr(eager, name).numpy(), err_msg=name)
    assert len(engine._GROUPED_GRAPHS) == 2


@pytest.mark.parametrize("T,takes", [(1000, True), (1601, True), (1602, False), (2000, False)])
def test_the_descent_takes_the_series_that_the_surface_takes(T, takes):
    """Length limits are checked on the host: a hierarchical fit is refused for
    the same series whether its voxels are many (descent) or few (surface)."""
    import ctypes as C

    from fastfuncstuff_gb300 import _lib

    lib, fake = _lib.load(), 256
    ld = (T + 63) // 64 * 64
    d = _lib.DescentArgs(V=100, T=T, K=5, P=545, n_designs=1, ld=ld, n_a=33, n_b=33, za=16, zb=16, ltop=4, n_groups=6,
                         n_list=49, n_rounds=2, n_cell_groups=500, n_chunks=40)
    n = lib.ffs_reml_descent_work_bytes(C.byref(d))
    assert (n > 0) == takes
    if not takes:
        assert "too long" in lib.ffs_last_error().decode()
        s = _lib.SurfaceArgs(V=100, T=T, K=5, P=545, p0=0, n_chunks=40, **{k: fake for k in (
            "yr_t", "coef", "logdet_R", "logdet_XtX", "proj", "chunk_start", "chunk_pairs", "surf", "crit0")})
        assert lib.ffs_reml_surface(C.byref(s), None) == _lib.FFS_ERR_INVALID
        assert "too long" in lib.ffs_last_error().decode()
    d.T, d.ld = 100, 128
    assert lib.ffs_reml_descent_work_bytes(C.byref(d)) > 0  # leaves no message behind


@gpu
@pytest.mark.parametrize("path", ["surface", "descent", "grouped", "global"])
def test_a_wait_that_ran_out_in_the_search_is_reported(path, monkeypatch):
    """The projection kernels leave at once when their flag is set, as they do
    after a wait that ran out: results for the host raise, and the descent's
    criterion on the device is a NaN."""
    from fastfuncstuff_gb300 import fit_glm_arma11, fit_glm_arma11_grouped
    from fastfuncstuff_gb300.glm import engine

    Y, X, _ = arma_data(5, 300, 90, 4)
    ax = np.linspace(-0.8, 0.8, 33)
    kw = dict(a_grid=ax, b_grid=ax, device=DEV, verbose=False)
    monkeypatch.setattr(engine, "DESCENT_MIN_WORK", 1 << 60 if path == "surface" else 0)

    def fit(**more):
        if path == "grouped":
            return fit_glm_arma11_grouped(Y, {0: X, 1: X[::-1].copy()}, np.arange(300) % 2, tr=2.0, cuda_graphs=False,
                                          **kw, **more)
        return fit_glm_arma11(Y, X, tr=2.0, estimate_per_voxel=path != "global", **kw, **more)

    assert torch.isfinite(fit().reml_likelihood).all()
    real = torch.zeros

    def preset(*size, **k):
        return real(*size, **k).fill_(1) if size == (1,) and k.get("dtype") is torch.int32 else real(*size, **k)

    monkeypatch.setattr(engine.torch, "zeros", preset)
    with pytest.raises(RuntimeError, match="bounded wait"):
        fit()
    if path in ("descent", "grouped"):
        assert torch.isnan(fit(return_device=True).reml_likelihood).all()


def test_small_batches_are_not_split_by_the_free_memory(monkeypatch):
    """The free memory decides the batch only where it is large: a fit of a few
    hundred voxels does not ask for it."""
    from fastfuncstuff_gb300.glm import arma

    asked = []
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda d=None: (asked.append(d), (1 << 28, 1 << 30))[1])
    assert arma._batch_size(200, 200, 117, 8, None, DEV) == 200 and not asked
    assert arma._batch_size(0, 200, 117, 8, None, DEV) == 1 and not asked
    assert arma._batch_size(200, 200, 117, 8, 64, DEV) == 64 and not asked
    per_voxel = 4 * (3 * 545 + 6 * 400 + 4 * 20 + 16)
    assert arma._batch_size(200_000, 400, 545, 20, None, DEV) == (1 << 27) // per_voxel and len(asked) == 1


@gpu
@pytest.mark.parametrize("T", [3, 130])
def test_prep_writes_splits_that_start_between_eight_byte_words(T):
    """The fp16 splits into buffers on 4-byte boundaries equal those on 8-byte
    ones (stored by narrower words)."""
    import ctypes as C

    from fastfuncstuff_gb300 import _lib

    V, ld = 37, (T + 7) // 8 * 8
    Y = torch.randn(V, T, device=DEV)
    scale, yexp = torch.empty(V, device=DEV), torch.empty(V, dtype=torch.int32, device=DEV)
    out = []
    for off in (0, 2):
        hi, lo = (torch.full((V * ld + 8,), 77, dtype=torch.int16, device=DEV) for _ in range(2))
        a = _lib.PrepArgs(V=V, T=T, K=0, Y=Y.data_ptr(), do_scale=1, center=0, ld_y=ld, scale=scale.data_ptr(),
                          yr_hi=hi.data_ptr() + 2 * off, yr_lo=lo.data_ptr() + 2 * off, yexp=yexp.data_ptr())
        _lib.check(_lib.load().ffs_reml_prep(C.byref(a), torch.cuda.current_stream().cuda_stream), "ffs_reml_prep")
        torch.cuda.synchronize()
        assert all((x[:off] == 77).all() and (x[off + V * ld :] == 77).all() for x in (hi, lo))
        out.append(torch.stack([hi[off : off + V * ld], lo[off : off + V * ld]]))
    assert torch.equal(out[0], out[1])


@gpu
def test_descent_scales_the_voxels_as_the_surface_does(monkeypatch):
    """The voxel scales of both searches bit for bit, of zero, constant, huge and NaN series too."""
    from fastfuncstuff_gb300.glm import engine

    V, T, K = 260, 130, 7
    Y, X, starts = arma_data(7, V, T, K, 2, baseline=50.0)
    Y[3], Y[17], Y[40], Y[41, 5] = 0.0, 12.5, Y[40] * 1e18, np.nan
    ax = torch.linspace(-0.8, 0.8, 33)
    Yd = torch.from_numpy(Y).to(DEV)
    f = engine.build_factors(torch.from_numpy(X).to(DEV), G.make_grid(ax, ax), G.run_layout(T, starts))
    monkeypatch.setattr(engine, "DESCENT_MIN_WORK", 0)
    assert engine._descent_plan(f, V) is not None
    got, want = engine.search(Yd, f), engine.search(Yd, f, keep_surface=True)
    assert torch.equal(got.scale.view(torch.int32), want.scale.view(torch.int32))


@pytest.mark.parametrize("a_max,corcut,lags", [(0.3, 1e-2, 16), (0.8, 1e-4, 48), (0.8, 1e-12, 128)])
def test_bands_of_the_banded_tests_reach_their_register_history(a_max, corcut, lags):
    """The grids that the banded GLS and surface tests use take the history of
    16, 48 and 128 lags that they are written for."""
    G.set_afni_mode(True, corcut)
    try:
        band = int(G.make_grid(torch.linspace(0.0, a_max, 4), torch.linspace(-0.4, 0.4, 5)).band.max())
    finally:
        G.set_afni_mode(False)
    assert {16: 0, 48: 16, 128: 48}[lags] < band <= lags


def test_builds_of_more_keys_than_the_descent_holds_keep_the_surface():
    """(design, pair) keys share a word with a slot in the descent's lists; a
    build of more of them is searched over the surface, which has no such limit."""
    import types

    from fastfuncstuff_gb300.glm import engine

    ax = torch.linspace(-0.8, 0.8, 33)
    g = G.make_grid(ax, ax)
    f = types.SimpleNamespace(U_hi=0, band_coef=None, P=g.P, T=100, K=5, grid=g, coef=torch.zeros(1))
    for n, takes in (((1 << 24) // g.P, True), ((1 << 24) // g.P + 1, False)):
        f.n_designs = n
        assert (engine._descent_plan(f, 1_000_000) is not None) == takes


@pytest.mark.parametrize("K,D,work", [(8, 1, 2.24e9), (14, 1, 1.68e9), (20, 1, 1.34e9), (30, 1, 1.01e9), (100, 1, 3.66e8),
                                      (130, 1, 3.66e8), (14, 4, 6.0e8), (100, 4, 6.0e8)])
def test_work_from_which_a_search_takes_the_descent(K, D, work):
    """Voxels x pairs x samples from which the descent is chosen: by the columns
    for one design, whose small fits wait for the host, and a fixed line for
    grouped ones."""
    import types

    from fastfuncstuff_gb300.glm import engine

    ax = torch.linspace(-0.8, 0.8, 33)
    g = G.make_grid(ax, ax)
    f = types.SimpleNamespace(U_hi=0, band_coef=None, P=g.P, T=400, K=K, grid=g, coef=torch.zeros(1), n_designs=D)
    for share, takes in ((0.98, False), (1.02, True)):
        assert (engine._descent_plan(f, int(share * work / (g.P * 400))) is not None) == takes
