"""The fixed-point kernels at the shapes of their launches: one row and one time
that stay in the form, calls large enough for a thread a row (more than four
waves of blocks) with one and two tiles of epochs, and orbits on both sides of
the lines where doubles are the more exact.

Tolerances: the path's flat 1e-9 max(1, |lnL|) for ln L, whatever e; 1e-9 of a
row's largest entry for the posterior and of K for a curve, with e <= 1/2, where
the column's (1 - e)^-2 is at most 4."""
import numpy as np
import pytest
import torch

from gpu_util import oracle_lnl, synth_chunk, synth_star
from test_gpu_posterior_edges import _expected

pytestmark = pytest.mark.gpu

MANY = 480_000


def _rows(rng, n, jitter, e_max=0.5):
    chunk = synth_chunk(rng, n, P_max=60.0, jitter=jitter)
    chunk[:, 1] = np.minimum(chunk[:, 1], e_max)
    return chunk


@pytest.mark.parametrize("jitter", [False, True])
@pytest.mark.parametrize("n,N,poly", [(1, 1, 1), (1, 20, 2), (33, 40, 1), (MANY, 20, 1),
                                      (MANY, 257, 1)])
def test_rows(cuda, n, N, poly, jitter):
    from thejoker_gb300 import device as dev
    rng = np.random.default_rng(n + N)
    star = synth_star(rng, N, poly=poly, t0=0.0, base=100.0)
    chunk = _rows(rng, n, jitter)
    table = dev.StarTable([star], jitter="applied" if jitter else "reference")
    cache = dev.PriorCache.from_samples(chunk)
    out = torch.empty((1, n), dtype=torch.float64, device="cuda")
    dev.lnl(table, cache, out, precision="fp64")
    a, A, l2 = (v.cpu().numpy() for v in dev.linear_posterior(table, cache, 0))
    pick = np.arange(n) if n < 1000 else np.concatenate(
        [np.arange(60), rng.integers(0, n, 80), np.arange(n - 60, n)])
    some = np.ascontiguousarray(chunk[pick])
    ref, got = oracle_lnl(star, some, jitter), out[0].cpu().numpy()
    assert np.all(np.abs(got[pick] - ref) <= 1e-9 * np.maximum(1.0, np.abs(ref)))
    assert np.all(np.isfinite(got))
    ea, eA = _expected(star, some, jitter)
    assert np.all(np.abs(a[pick] - ea).max(1) <= 1e-9 * np.maximum(1.0, np.abs(ea).max(1)))
    assert np.all(np.abs(A[pick] - eA).max((1, 2)) <= 1e-9 * np.abs(eA).max((1, 2)))
    free = dict(star, k_prior=np.array([1.0, 30.0, 365.25, 1e12]))         # unclipped
    ref = oracle_lnl(free, some, jitter)
    assert np.all(np.abs(l2[pick] - ref) <= 1e-9 * np.maximum(1.0, np.abs(ref)))


@pytest.mark.parametrize("rows,times", [(1, 1), (1, 5), (2, 40)])
def test_curves(cuda, rows, times):
    from thejoker_gb300 import device as dev
    from thejoker_gb300.linear import rv_unit_columns
    rng = np.random.default_rng(rows + times)
    c = _rows(rng, rows, False)
    K = rng.uniform(1.0, 50.0, rows)
    t = 2456000.0 + rng.uniform(100.0, 200.0, times)
    el = np.stack([c[:, 0], K, c[:, 1], c[:, 2], c[:, 3]], 1)
    got = dev.rv_from_elements(torch.from_numpy(t).cuda(), torch.from_numpy(el).cuda(), 2456000.0)
    want = K[:, None] * rv_unit_columns(t, 2456000.0, c[:, 0], c[:, 1], c[:, 2], c[:, 3])
    assert np.all(np.abs(got.cpu().numpy() - want) <= 1e-9 * K[:, None])


@pytest.mark.parametrize("jitter", [False, True])
@pytest.mark.parametrize("ratio", [0.4, 0.9, 1.1, 2.2, 4.4, 9.0, 100.0])
def test_long_periods(cuda, ratio, jitter):
    """Periods of `ratio` spans, eccentricities around each of the lines."""
    rng = np.random.default_rng(int(10 * ratio))
    star = synth_star(rng, 20, t0=0.0, base=100.0)
    span = np.ptp(star["t"])
    chunk = synth_chunk(rng, 64, jitter=jitter)
    chunk[:, 0] = ratio * span * rng.uniform(0.98, 1.02, 64)
    chunk[:, 1] = np.tile([0.3, 0.874, 0.876, 0.984, 0.985, 0.998, 0.9989, 0.9995], 8)
    from thejoker_gb300 import device as dev
    table = dev.StarTable([star], jitter="applied" if jitter else "reference")
    out = torch.empty((1, 64), dtype=torch.float64, device="cuda")
    dev.lnl(table, dev.PriorCache.from_samples(chunk), out, precision="fp64")
    ref = oracle_lnl(star, chunk, jitter)
    assert np.all(np.abs(out[0].cpu().numpy() - ref) <= 1e-9 * np.maximum(1.0, np.abs(ref)))
