"""Routes of the host-facing calls that depend on their sizes: the drop-in's
mapped pinned rows, columns of a JokerSamples uploaded as they are, and the
batched restart of an iterative handle.  Each against the route beside it; the
results are the same numbers."""
import numpy as np
import pytest
import torch

from gpu_util import synth_chunk, synth_star

pytestmark = pytest.mark.gpu


def _setup(N, seed=3):
    from thejoker_gb300 import JokerPrior, RVData
    star = synth_star(np.random.default_rng(seed), N)
    prior = JokerPrior.default(P_min=2.0, P_max=1024.0, sigma_K0=30.0, sigma_v=100.0)
    return RVData(star["t"], star["rv"], 1.0 / np.sqrt(star["ivar"])), prior


@pytest.mark.parametrize("rows", [1, 31, 16384, 16385])
def test_mapped_rows(cuda, rows):
    from thejoker_gb300 import GPUJokerHelper
    from thejoker_gb300.data import validate_prepare_data
    data, prior = _setup(7)
    all_data, _, trend = validate_prepare_data(data, 1, 0)
    helper = GPUJokerHelper(all_data, prior, trend)
    chunk = synth_chunk(np.random.default_rng(rows), rows)
    want = helper.batch_marginal_ln_likelihood_device(torch.from_numpy(chunk).cuda())
    got = helper.batch_marginal_ln_likelihood(chunk)
    np.testing.assert_array_equal(got, want.cpu().numpy())
    assert got.flags.writeable


@pytest.mark.parametrize("in_memory", [True, False])
def test_columns_and_rows(cuda, in_memory):
    """Columns with strides and read-only ones, against the packed rows."""
    from thejoker_gb300 import JokerSamples, TheJoker
    data, prior = _setup(9)
    chunk = synth_chunk(np.random.default_rng(4), 5001)
    frozen = np.ascontiguousarray(chunk[:, 3])
    frozen.flags.writeable = False
    table = JokerSamples({"P": chunk[:, 0], "e": chunk[::-1, 1][::-1], "omega": chunk[:, 2],
                          "M0": frozen, "s": chunk[:, 4]})
    out = []
    for samples in (table, chunk) if in_memory else (table, JokerSamples(
            dict(zip(("P", "e", "omega", "M0", "s"), chunk.T.copy())))):
        joker = TheJoker(prior, rng=np.random.default_rng(11))
        out.append(joker.rejection_sample(data, samples, in_memory=in_memory,
                                          return_all_logprobs=True))
    (a, la), (b, lb) = out
    np.testing.assert_array_equal(la, lb)
    for k in a.keys():
        np.testing.assert_array_equal(a[k], b[k])


@pytest.mark.parametrize("stars", [1, 101])
def test_restart(cuda, stars):
    from thejoker_gb300 import device as dev
    from thejoker_gb300.iterative import IterativeBatch
    rng = np.random.default_rng(stars)
    table = dev.StarTable([synth_star(rng, int(n)) for n in rng.integers(3, 12, stars)])
    cache = dev.PriorCache.from_samples(synth_chunk(rng, 20_000))
    seeds = list(range(stars))
    engine = IterativeBatch(table, cache, 16, seeds=[s + 1000 for s in seeds]).run()
    got = engine.reset(seeds).run().results()
    want = IterativeBatch(table, cache, 16, seeds=seeds).run().results()
    np.testing.assert_array_equal(got[0], want[0])
    for g, w in zip(got[1], want[1]):
        np.testing.assert_array_equal(g, w)
