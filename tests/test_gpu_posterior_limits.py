"""joker_linear_posterior at the ends of the K prior's range: variances near the
largest double and beyond it, against the matrix formulas with 1/Lambda0 in
place of Lambda0.

Tolerance: that of the posterior against the matrix formulas, 1e-9 of a row's
largest entry; e <= 0.9, where (1 - e)^-2 allows for the column.  ln L adds the
logarithm of Lambda0, which is exact to an ulp of its value."""
import numpy as np
import pytest
import torch

from gpu_util import synth_chunk, synth_star

pytestmark = pytest.mark.gpu


def _expected(star, chunk, lam0, jitter):
    """a, A and ln L for K prior variances lam0 (one per row, inf allowed)."""
    from thejoker_gb300.linear import rv_unit_columns
    m = rv_unit_columns(star["t"], star["t_ref"], chunk[:, 0], chunk[:, 1], chunk[:, 2],
                        chunk[:, 3])
    y, a, A, lnl = star["rv"], [], [], []
    for k, s in enumerate(chunk[:, 4]):
        M = np.vstack([m[k][None], star["trend_M"].T])
        w = star["ivar"] / (1 + s * s * star["ivar"]) if jitter else star["ivar"]
        inv_lam = np.append(1 / lam0[k], 1 / star["lam"][1:])
        G = (M * w) @ M.T + np.diag(inv_lam)
        d = 1 / np.sqrt(np.diag(G))
        inv = np.linalg.inv(G * d[:, None] * d[None]) * d[:, None] * d[None]
        q = (M * w) @ y
        a.append(inv @ q)
        A.append(inv)
        logdet = np.linalg.slogdet(G * d[:, None] * d[None])[1] - 2 * np.log(d).sum()
        lnl.append(-0.5 * ((w * y * y).sum() - q @ inv @ q + len(y) * np.log(2 * np.pi) -
                           np.log(w).sum() + np.log(lam0[k]) + np.log(star["lam"][1:]).sum() +
                           logdet))
    return np.array(a), np.array(A), np.array(lnl)


def _posterior(star, chunk, jitter):
    from thejoker_gb300 import device as dev
    table = dev.StarTable([star], jitter="applied" if jitter else "reference")
    cache = dev.PriorCache.from_samples(chunk)
    return [v.cpu().numpy() for v in dev.linear_posterior(table, cache, 0)]


@pytest.mark.parametrize("jitter", [False, True])
@pytest.mark.parametrize("lam0", [1e290, 1e303, 1e307, np.inf])
@pytest.mark.parametrize("poly", [1, 2])
def test_wide_prior(cuda, lam0, poly, jitter):
    rng = np.random.default_rng(17)
    star = synth_star(rng, 20, poly=poly, t0=0.0, base=100.0)
    chunk = synth_chunk(rng, 65, P_max=60.0, jitter=jitter)
    chunk[:, 1] = np.minimum(chunk[:, 1], 0.9)
    if np.isfinite(lam0):
        star["k_prior"], star["lam"][0] = np.zeros(4), lam0
    else:                                    # the scaled variance overflows
        star["k_prior"] = np.array([1.0, 1e160, 365.25, 500.0])
    a, A, lnl = _posterior(star, chunk, jitter)
    ea, eA, el = _expected(star, chunk, np.full(len(chunk), lam0), jitter)
    grow = (1.0 - chunk[:, 1]) ** -2
    assert np.all(np.abs(a - ea).max(1) <= 1e-9 * grow * np.maximum(1.0, np.abs(ea).max(1)))
    assert np.all(np.abs(A - eA).max((1, 2)) <= 1e-9 * grow * np.abs(eA).max((1, 2)))
    if np.isfinite(lam0):
        assert np.all(np.abs(lnl - el) <= 1e-9 * grow * np.maximum(1.0, np.abs(el)))
    else:
        assert np.all(lnl == -np.inf)


@pytest.mark.parametrize("jitter", [False, True])
@pytest.mark.parametrize("N,poly", [(3, 1), (20, 2), (40, 1)])
def test_parabolic_row(cuda, N, poly, jitter):
    """e = 1: an infinite K prior variance; the unit-K column is the limit's, and
    the row is finite."""
    rng = np.random.default_rng(N)
    star = synth_star(rng, N, poly=poly, t0=0.0, base=100.0)
    chunk = synth_chunk(rng, 5, P_max=60.0, jitter=jitter)
    chunk[2, 1] = 1.0
    a, A, lnl = _posterior(star, chunk, jitter)
    assert np.all(np.isfinite(a)) and np.all(np.isfinite(A))
    assert lnl[2] == -np.inf and np.all(np.isfinite(np.delete(lnl, 2)))
