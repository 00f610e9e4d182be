"""A row's FP64 ln L does not depend on the call it is in: few rows (four warps
share the epochs), many (one thread takes them), the refinement's list (a warp a
row) and what overflows it (a thread a row, epochs from global memory) give the
same number, bit for bit, with and without the jitter: the fixed-point form's
rows.  The warp form in doubles sums in another order (a few ulps of ln L); a star
of one epoch, whose time scale is zero, has such rows beyond e = 7/8."""
import numpy as np
import pytest
import torch

from gpu_util import synth_chunk, synth_star

pytestmark = pytest.mark.gpu


def _fp64(table, chunk):
    from thejoker_gb300 import device as dev
    out = torch.empty((1, len(chunk)), dtype=torch.float64, device="cuda")
    dev.lnl(table, dev.PriorCache.from_samples(chunk), out, precision="fp64")
    return out[0].cpu().numpy()


@pytest.mark.parametrize("jitter", [False, True])
@pytest.mark.parametrize("N,poly,noff", [(1, 1, 0), (3, 1, 0), (16, 1, 0), (37, 2, 0),
                                         (67, 3, 1), (258, 1, 0)])
def test_same_number(cuda, N, poly, noff, jitter):
    from thejoker_gb300 import device as dev
    rng = np.random.default_rng(N)
    star = synth_star(rng, N, poly=poly, noff=noff, t0=0.0, base=100.0)
    table = dev.StarTable([star], jitter="applied" if jitter else "reference")
    n = 1 << 20                                        # more than four waves of any kernel
    chunk = synth_chunk(rng, n, P_max=60.0, jitter=jitter)
    many = _fp64(table, chunk)
    few = np.concatenate([_fp64(table, np.ascontiguousarray(chunk[a:a + 500]))
                          for a in (0, n // 2, n - 500)])
    pick = np.concatenate([np.arange(a, a + 500) for a in (0, n // 2, n - 500)])
    np.testing.assert_array_equal(few, many[pick])
    # every row of a mixed ln L with an open bound is re-evaluated: the first
    # 65536 + 64 per 8192 rows through the list, the rest beside it
    m = 140_000
    lnl = torch.full((m,), float(many[:m].max()), dtype=torch.float64, device="cuda")
    err = torch.full((m,), 1e30, dtype=torch.float32, device="cuda")
    top = dev.MaxKeys(1)
    one = torch.empty((1, m), dtype=torch.float64, device="cuda")
    cache = dev.PriorCache.from_samples(chunk[:m])
    dev.lnl(table, cache, one, precision="fp64", max_keys=top)
    done = dev.refine_band(table, cache, lnl, err, top,
                           [dict(lnl_off=0, n=m, out_off=0, max_out=0, max_slot=0, star=0,
                                 row0=0)])
    assert int(done.item()) == m
    got, fixed = lnl.cpu().numpy(), chunk[:m, 1] <= (0.875 if N == 1 else 0.999)
    np.testing.assert_array_equal(got[fixed], many[:m][fixed])
    np.testing.assert_allclose(got, many[:m], rtol=64 * 2.0 ** -53)
