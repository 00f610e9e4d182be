"""HostRejection's slices shared by several stars at FP64 and with the jitter
applied, against the same stars over a device cache at FP64.  Sizes around the
ends of the first and second slice."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [(1 << 18) + 1, 3 * (1 << 18) + 33])
@pytest.mark.parametrize("jitter", ["reference", "applied"])
@pytest.mark.parametrize("precision", ["mixed_fast", "fp64"])
def test_shared_slices(cuda, rows, jitter, precision):
    from thejoker_gb300 import device as dev
    from thejoker_gb300.batch import BatchRejection
    from thejoker_gb300.pipeline import HostRejection, _shares
    from thejoker_gb300.synthetic import fill_prior_cache, survey_stars
    assert _shares(3, rows)
    stars = survey_stars(3, seed=6, n_max=24)
    chunk = fill_prior_cache(np.empty((rows, 5)), 4)
    chunk[:, 4] = np.exp(np.random.default_rng(1).normal(np.log(0.5), 1.0, rows))
    table = dev.StarTable(stars, jitter=jitter)
    hr = HostRejection(table, rows, precision=precision, max_out=300)
    seeds = [7, 8, 9]
    pcg = [dev.pcg64_state(np.random.default_rng(sd)) for sd in seeds]
    counts, idx = hr.run(torch.from_numpy(chunk).pin_memory(), pcg)
    cache = dev.PriorCache.from_samples(chunk)
    c64, i64, _ = BatchRejection(stars, cache, precision="fp64", jitter=jitter, max_out=300,
                                 seeds=seeds).run().results()
    np.testing.assert_array_equal(counts, c64)
    for k in range(3):
        np.testing.assert_array_equal(idx[k], i64[k])
