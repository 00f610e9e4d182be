"""A captured joker_linear_posterior launch on a slot table, replayed after the
slot was given another star: every property of the star (a K prior mean, weights
without a fixed-point form) is the device's, not the one at capture.

Tolerance: that of the posterior against the matrix formulas, 1e-9 of a row's
largest entry; e <= 0.9, where (1 - e)^-2 allows for the column."""
import numpy as np
import pytest
import torch

from gpu_util import oracle_lnl, synth_chunk, synth_star
from test_gpu_posterior_edges import _expected

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jitter", [False, True])
def test_replay_after_set(cuda, jitter):
    from thejoker_gb300 import device as dev
    rng = np.random.default_rng(31)
    stars = [synth_star(rng, N, t0=0.0, base=100.0) for N in (20, 18, 16)]
    stars[1]["mu"][0] = 3.0
    stars[2]["ivar"] = stars[2]["ivar"] * np.where(np.arange(16) % 2, 1e-3, 1.0)
    chunk = synth_chunk(rng, 70, P_max=60.0, jitter=jitter)
    chunk[:, 1] = np.minimum(chunk[:, 1], 0.9)
    table = dev.StarTable.slots(2, 20, 2, jitter="applied" if jitter else "reference")
    cache = dev.PriorCache.from_samples(chunk)
    rows = torch.arange(len(chunk), device="cuda")
    table.set(1, stars[0])
    dev.linear_posterior(table, cache, 1, rows)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = dev.linear_posterior(table, cache, 1, rows)
    grow = (1.0 - chunk[:, 1]) ** -2
    for star in stars:
        table.set(1, star)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        a, A, lnl = (v.cpu().numpy() for v in out)
        ea, eA = _expected(star, chunk, jitter)
        assert np.all(np.abs(a - ea).max(1) <= 1e-9 * grow * np.maximum(1.0, np.abs(ea).max(1)))
        assert np.all(np.abs(A - eA).max((1, 2)) <= 1e-9 * grow * np.abs(eA).max((1, 2)))
        free = dict(star, k_prior=np.array([1.0, 30.0, 365.25, 1e12]))     # unclipped
        ref = oracle_lnl(free, chunk, jitter)
        assert np.all(np.abs(lnl - ref) <= 1e-9 * grow * np.maximum(1.0, np.abs(ref)))
