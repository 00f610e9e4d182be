"""FP64 ln L of stars without the fixed-point form, alone and beside stars that
have it: around one block's rows and one and two tiles of epochs, against the
CPU oracle.  Tolerance: the path's 1e-9 max(1, |lnL|); e <= 0.9."""
import numpy as np
import pytest
import torch

from gpu_util import oracle_lnl, synth_chunk, synth_star

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jitter", [False, True])
@pytest.mark.parametrize("S,N,poly,noff", [(1, 2, 1, 0), (127, 16, 1, 0), (128, 17, 2, 0),
                                           (129, 256, 3, 1), (300, 257, 1, 0)])
@pytest.mark.parametrize("stars", ["alone", "beside"])
def test_doubles(cuda, S, N, poly, noff, jitter, stars):
    from thejoker_gb300 import device as dev
    rng = np.random.default_rng(S + N)
    # (a baseline of 100 days: a quadratic trend in double precision)
    group = [synth_star(rng, n, poly=poly, noff=noff, t0=0.0, base=100.0) for n in (N, 7, N + 1)]
    for star in group[::2] if stars == "beside" else group:
        star["ivar"] = star["ivar"] * np.where(np.arange(len(star["t"])) % 2, 1e-3, 1.0)
    chunk = synth_chunk(rng, S, P_max=60.0, jitter=jitter)
    chunk[:, 1] = np.minimum(chunk[:, 1], 0.9)
    table = dev.StarTable(group, jitter="applied" if jitter else "reference")
    cache = dev.PriorCache.from_samples(chunk)
    out = torch.empty((3, S), dtype=torch.float64, device="cuda")
    keys = dev.MaxKeys(3)
    dev.lnl(table, cache, out, precision="fp64", max_keys=keys)
    one = torch.empty((1, S), dtype=torch.float64, device="cuda")
    dev.lnl(table, cache, one, precision="fp64", star0=2, n_sel=1)
    got = out.cpu().numpy()
    for k, star in enumerate(group):
        ref = oracle_lnl(star, chunk, jitter)
        assert np.all(np.abs(got[k] - ref) <= 1e-9 * np.maximum(1.0, np.abs(ref)))
    np.testing.assert_array_equal(keys.values(), got.max(1))
    ref = oracle_lnl(group[2], chunk, jitter)
    assert np.all(np.abs(one[0].cpu().numpy() - ref) <= 1e-9 * np.maximum(1.0, np.abs(ref)))


@pytest.mark.parametrize("jitter", [False, True])
@pytest.mark.parametrize("rows", [12 * 152 * 128 - 1, 12 * 152 * 128 + 1])
def test_block_sizes(cuda, rows, jitter):
    """Both sides of the line between blocks of one warp and of four: rows at
    both ends and in between against the oracle."""
    from thejoker_gb300 import device as dev
    rng = np.random.default_rng(rows)
    star = synth_star(rng, 5, t0=0.0, base=100.0)
    star["ivar"] = star["ivar"] * np.where(np.arange(5) % 2, 1e-3, 1.0)
    chunk = synth_chunk(rng, rows, P_max=60.0, jitter=jitter)
    chunk[:, 1] = np.minimum(chunk[:, 1], 0.9)
    table = dev.StarTable([star], jitter="applied" if jitter else "reference")
    out = torch.empty((1, rows), dtype=torch.float64, device="cuda")
    dev.lnl(table, dev.PriorCache.from_samples(chunk), out, precision="fp64")
    pick = np.concatenate([np.arange(140), rng.integers(0, rows, 100),
                           np.arange(rows - 140, rows)])
    got, ref = out[0].cpu().numpy(), oracle_lnl(star, np.ascontiguousarray(chunk[pick]), jitter)
    assert np.all(np.abs(got[pick] - ref) <= 1e-9 * np.maximum(1.0, np.abs(ref)))
    assert np.all(np.isfinite(got))
