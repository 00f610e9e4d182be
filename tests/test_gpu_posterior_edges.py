"""joker_linear_posterior at the edges of its block shapes (one sample, a part
of a block, more than a block; fewer and more epochs than are shared out or
staged at once), for rows that the fixed-point form hands over, and for stars
without that form, against the matrix formulas in 64 bits.

Tolerance: 1e-9 of the largest entry of the row, times (1 - e)^-2 for the
column near pericentre; the ln L tolerance is the likelihood's."""
import numpy as np
import pytest
import torch

from gpu_util import oracle_lnl, synth_chunk, synth_star

pytestmark = pytest.mark.gpu


def _expected(star, chunk, jitter):
    from thejoker_gb300.linear import rv_unit_columns
    m = rv_unit_columns(star["t"], star["t_ref"], chunk[:, 0], chunk[:, 1], chunk[:, 2],
                        chunk[:, 3])
    L = 1 + star["trend_M"].shape[1]
    a, A = [], []
    for k, (P, e, _, _, s) in enumerate(chunk):
        M = np.vstack([m[k][None], star["trend_M"].T])
        w = star["ivar"] / (1 + s * s * star["ivar"]) if jitter else star["ivar"]
        lam = star["lam"].copy()
        lam[0] = star["k_prior"][1] ** 2 / (1 - e * e) * (P / star["k_prior"][2]) ** (-2 / 3)
        G = (M * w) @ M.T + np.diag(1 / lam)
        d = 1 / np.sqrt(np.diag(G))
        inv = np.linalg.inv(G * d[:, None] * d[None]) * d[:, None] * d[None]
        A.append(inv)
        a.append(star["mu"] + inv @ ((M * w) @ (star["rv"] - star["mu"] @ M)))
    return np.array(a).reshape(-1, L), np.array(A)


@pytest.mark.parametrize("jitter", [False, True])
@pytest.mark.parametrize("n,N,poly,noff", [(1, 1, 1, 0), (33, 15, 1, 0), (129, 16, 2, 1),
                                           (65, 257, 3, 0)])
@pytest.mark.parametrize("form", ["fixed", "weights", "mean"])
def test_posterior_edges(cuda, n, N, poly, noff, jitter, form):
    from thejoker_gb300 import device as dev
    rng = np.random.default_rng(n + N)
    star = synth_star(rng, N, poly=poly, noff=noff, t0=0.0, base=100.0)
    if form == "weights":
        star["ivar"] = star["ivar"] * np.where(np.arange(N) % 2, 1e-3, 1.0)
    if form == "mean":
        star["mu"][0] = 3.0
    chunk = synth_chunk(rng, n, P_max=60.0, jitter=jitter)
    chunk[:, 1] = np.minimum(chunk[:, 1], 0.9)
    chunk[n // 2, 1] = 0.9995
    table = dev.StarTable([star], jitter="applied" if jitter else "reference")
    cache = dev.PriorCache.from_samples(chunk)
    rows = torch.from_numpy(rng.permutation(n)).cuda()
    a, A, lnl = (v.cpu().numpy() for v in dev.linear_posterior(table, cache, 0, rows))
    picked = chunk[rows.cpu().numpy()]
    ea, eA = _expected(star, picked, jitter)
    grow = (1.0 - picked[:, 1]) ** -2
    assert np.all(np.abs(a - ea).max(1) <= 1e-9 * grow * np.maximum(1.0, np.abs(ea).max(1)))
    assert np.all(np.abs(A - eA).max((1, 2)) <= 1e-9 * grow * np.abs(eA).max((1, 2)))
    star = dict(star, k_prior=np.array([1.0, 30.0, 365.25, 1e12]))     # unclipped
    ref = oracle_lnl(star, picked, jitter)
    assert np.all(np.abs(lnl - ref) <= 1e-9 * grow * np.maximum(1.0, np.abs(ref)))
