"""The fixed-point form of the FP64 path at the edges of its range, against the
CPU oracle.  Tolerance: the path's 1e-9 max(1, |lnL|), times (1 - e)^-2, by
which both sides' column errors grow near pericentre."""
import numpy as np
import pytest
import torch

from gpu_util import oracle_lnl, synth_chunk, synth_star

pytestmark = pytest.mark.gpu


def _lnl(star, chunk, jitter):
    from thejoker_gb300 import device as dev
    table = dev.StarTable([star], jitter="applied" if jitter else "reference")
    cache = dev.PriorCache.from_samples(chunk)
    out = torch.empty((1, len(chunk)), dtype=torch.float64, device="cuda")
    dev.lnl(table, cache, out, precision="fp64")
    return out[0].cpu().numpy()


def _check(star, chunk, jitter):
    got, ref = _lnl(star, chunk, jitter), oracle_lnl(star, chunk, jitter)
    tol = 1e-9 * np.maximum(1.0, np.abs(ref)) / (1.0 - chunk[:, 1]) ** 2
    assert np.all(np.abs(got - ref) <= tol)


@pytest.mark.parametrize("jitter", [False, True])
@pytest.mark.parametrize("N,poly,noff", [(1, 1, 0), (3, 1, 0), (33, 2, 1), (256, 1, 0),
                                         (257, 3, 1), (530, 2, 0), (40, 3, 2)])
def test_epochs_and_columns(cuda, N, poly, noff, jitter):
    rng = np.random.default_rng(100 * N + poly)
    star = synth_star(rng, N, poly=poly, noff=min(noff, 1), t0=0.0)
    if noff == 2:                            # six linear parameters
        star["trend_M"] = np.hstack([star["trend_M"], (star["t"] > 500.0)[:, None] * 1.0])
        star["mu"], star["lam"] = np.zeros(6), np.append(star["lam"], 4.0)
    chunk = synth_chunk(rng, 129 if N < 100 else 12, jitter=jitter)
    chunk[:, 1] = np.minimum(chunk[:, 1], 0.9)
    _check(star, chunk, jitter)


@pytest.mark.parametrize("jitter", [False, True])
def test_sample_edges(cuda, jitter):
    """Eccentricities and jitters on both sides of the lines, tiny and huge
    periods, angles of either sign, times before the reference."""
    rng = np.random.default_rng(7)
    star = synth_star(rng, 20, t0=0.0)
    star["t_ref"] = 400.0
    chunk = synth_chunk(rng, 96, jitter=jitter)
    chunk[:, 1] = np.minimum(chunk[:, 1], 0.9)
    chunk[:8, 1] = [0.0, 1e-300, 1e-9, 3e-6, 0.99, 0.999, 0.99900001, 0.9995]
    chunk[8:12, 0] = [1e-3, 1e5, 1e9, 2.0 ** -22]
    chunk[12:16, 3] = [-3.0, 40.0, 0.0, 2000.0]
    chunk[16:20, 2] = [-3.0, 40.0, 0.0, 2000.0]
    if jitter:
        chunk[20:26, 4] = [0.0, 1e-8, 1e2, 1e5, 2e5, 1e9]
    phase = np.abs(1000.0 / chunk[:, 0])     # turns: a double's phase is good to 2^-52 of them
    keep = phase < 1e6
    got, ref = _lnl(star, chunk, jitter), oracle_lnl(star, chunk, jitter)
    tol = 1e-9 * np.maximum(1.0, np.abs(ref)) / (1.0 - chunk[:, 1]) ** 2
    assert np.all((np.abs(got - ref) <= tol)[keep]) and np.all(np.isfinite(got))


@pytest.mark.parametrize("ratio", [255.0, 257.0, 1e8])
@pytest.mark.parametrize("jitter", [False, True])
def test_weight_spans(cuda, ratio, jitter):
    rng = np.random.default_rng(8)
    star = synth_star(rng, 12, poly=2, t0=0.0)
    star["ivar"] = 1.0 / np.geomspace(1.0, ratio, 12)
    chunk = synth_chunk(rng, 64, jitter=jitter)
    chunk[:, 1] = np.minimum(chunk[:, 1], 0.9)
    _check(star, chunk, jitter)


def test_prior_mean(cuda):
    """A K prior mean other than zero: the jitter form runs in doubles."""
    rng = np.random.default_rng(9)
    star = synth_star(rng, 12, t0=0.0)
    star["mu"] = np.array([5.0, 1.0])
    for jitter in (False, True):
        chunk = synth_chunk(rng, 64, jitter=jitter)
        chunk[:, 1] = np.minimum(chunk[:, 1], 0.9)
        _check(star, chunk, jitter)


@pytest.mark.parametrize("rows,times", [(1, 1), (3, 7), (2, 255), (5, 256), (33, 257), (2, 1001)])
def test_rv_curves(cuda, rows, times):
    """Curves that end inside, at and beyond a warp's share of times, times on
    both sides of t0, and one orbit beyond the fixed-point form."""
    from thejoker_gb300 import device as dev
    from thejoker_gb300.linear import rv_unit_columns
    rng = np.random.default_rng(rows * 10000 + times)
    c = synth_chunk(rng, rows)
    c[:, 1] = np.minimum(c[:, 1], 0.9)
    c[-1, 1] = 0.9995
    K = rng.uniform(1.0, 50.0, rows)
    t, t0 = 2456000.0 + rng.uniform(0.0, 2000.0, times), 2456700.0
    el = np.stack([c[:, 0], K, c[:, 1], c[:, 2], c[:, 3]], 1)
    got = dev.rv_from_elements(torch.from_numpy(t).cuda(), torch.from_numpy(el).cuda(), t0)
    want = K[:, None] * rv_unit_columns(t, t0, c[:, 0], c[:, 1], c[:, 2], c[:, 3])
    tol = 1e-9 * K / (1.0 - c[:, 1]) ** 2
    assert np.all(np.abs(got.cpu().numpy() - want) <= tol[:, None])


@pytest.mark.parametrize("lo,hi", [(2.0, 1024.0), (2.0, 2.0000001), (1e-300, 1e300),
                                   (1e-310, 1e-300)])
def test_period_draws(cuda, lo, hi):
    """P = P_min (P_max / P_min)^u over narrow, ordinary and extreme ranges, the
    last through doubles; 60 ulps of exp's argument at 700."""
    from thejoker_gb300 import _native as nat
    from thejoker_gb300 import device as dev
    n, seed = 5000, 99
    packed = torch.empty((n, 5), dtype=torch.float64, device="cuda")
    dev.PriorCache(n).sample_prior(
        dict(P_min=lo, P_max=hi, e_alpha=0.867, e_beta=3.03, s_kind=nat.JOKER_S_FIXED,
             s_value=0.0), n, seed=seed, packed=packed)
    P = packed[:, 0].cpu().numpy()
    assert np.all((P >= lo * (1 - 1e-13)) & (P <= hi * (1 + 1e-13)))
    # the stream's first uniform: Philox4x32-10 of counter (g, 0, 0, tag)
    g = np.arange(n, dtype=np.uint64)
    c = [g, 0 * g, 0 * g, 0 * g + np.uint64(0x4A6F6B72)]
    k, low = [np.uint64(seed), np.uint64(0)], np.uint64(0xFFFFFFFF)
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ k[0], p1 & low, (p0 >> np.uint64(32)) ^ c[3] ^ k[1],
             p0 & low]
        k = [(k[0] + np.uint64(0x9E3779B9)) & low, (k[1] + np.uint64(0xBB67AE85)) & low]
    u = (((c[1] << np.uint64(32)) | c[0]) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53
    want = np.exp(np.log(lo) + u * (np.log(hi) - np.log(lo)))
    np.testing.assert_allclose(P, want, rtol=60 * 2.0 ** -53 * 700)


@pytest.mark.parametrize("mean", [np.nan, np.inf, -np.inf])
def test_prior_mean_not_finite(cuda, mean):
    """No finite velocity is left: NaN everywhere, as in doubles."""
    rng = np.random.default_rng(10)
    star = synth_star(rng, 12, t0=0.0)
    star["mu"] = np.array([0.0, mean])
    assert np.all(np.isnan(_lnl(star, synth_chunk(rng, 33), False)))
