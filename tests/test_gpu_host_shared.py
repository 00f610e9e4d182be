"""HostRejection with several stars: slices of the host chunk shared by them,
against the same stars' rows over a device cache at FP64.  Sizes around the
ends of the first and second slice and below where slices pay."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [209_715, 1 << 18, (1 << 18) + 1, 3 * (1 << 18) + 33])
@pytest.mark.parametrize("precision", ["mixed_fast", "mixed"])
def test_shared_slices(cuda, rows, precision):
    from thejoker_gb300 import device as dev
    from thejoker_gb300.batch import BatchRejection
    from thejoker_gb300.pipeline import HostRejection
    from thejoker_gb300.synthetic import fill_prior_cache, survey_stars
    stars = survey_stars(3, seed=5, n_max=24)
    chunk = fill_prior_cache(np.empty((rows, 5)), 3)
    table = dev.StarTable(stars)
    host = torch.from_numpy(chunk).pin_memory()
    hr = HostRejection(table, rows + 7 - rows % 2, precision=precision, max_out=300)
    cache = dev.PriorCache.from_samples(chunk)
    for seeds in ([1, 2, 3], [4, 5, 6]):                     # the buffers serve again
        pcg = [dev.pcg64_state(np.random.default_rng(sd)) for sd in seeds]
        counts, idx = hr.run(host, pcg)
        c64, i64, _ = BatchRejection(table, cache, precision="fp64", max_out=300,
                                     seeds=seeds).run().results()
        np.testing.assert_array_equal(counts, c64)
        for k in range(3):
            np.testing.assert_array_equal(idx[k], i64[k])
