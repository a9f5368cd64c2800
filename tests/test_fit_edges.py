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
