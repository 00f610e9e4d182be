"""joker_rv_from_elements for curves of few times, which take fewer lanes per
orbit: around one warp's, one block's and one grid pass's orbits, with orbits
that the fixed-point form hands over among their neighbours.

Tolerance: 1e-9 K, times (1 - e)^-2 by which both sides' column errors grow near
pericentre; e <= 0.9 but for the orbits handed over."""
import numpy as np
import pytest
import torch

from gpu_util import synth_chunk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("times", [1, 2, 7, 8, 9, 33])
@pytest.mark.parametrize("rows", [1, 3, 31, 129, 1025])
def test_short_curves(cuda, rows, times):
    from thejoker_gb300 import device as dev
    from thejoker_gb300.linear import rv_unit_columns
    rng = np.random.default_rng(rows * 100 + times)
    c = synth_chunk(rng, rows)
    c[:, 1] = np.minimum(c[:, 1], 0.9)
    if rows > 1:
        c[::7, 1] = 0.9995
    K = rng.uniform(1.0, 50.0, rows)
    t, t0 = 2456000.0 + rng.uniform(0.0, 2000.0, times), 2456700.0
    el = np.stack([c[:, 0], K, c[:, 1], c[:, 2], c[:, 3]], 1)
    got = dev.rv_from_elements(torch.from_numpy(t).cuda(), torch.from_numpy(el).cuda(), t0)
    want = K[:, None] * rv_unit_columns(t, t0, c[:, 0], c[:, 1], c[:, 2], c[:, 3])
    tol = 1e-9 * K / (1.0 - c[:, 1]) ** 2
    assert np.all(np.abs(got.cpu().numpy() - want) <= tol[:, None])


def test_many_orbits(cuda):
    """More orbits than one pass of the grid takes, one lane each."""
    from thejoker_gb300 import device as dev
    from thejoker_gb300.linear import rv_unit_columns
    rng = np.random.default_rng(8)
    n = 152 * 64 * 128 + 77
    c = synth_chunk(rng, n)
    c[:, 1] = np.minimum(c[:, 1], 0.9)
    el = np.stack([c[:, 0], np.ones(n), c[:, 1], c[:, 2], c[:, 3]], 1)
    t = torch.tensor([512.25], dtype=torch.float64, device="cuda")
    got = dev.rv_from_elements(t, torch.from_numpy(el).cuda(), 0.0)[:, 0].cpu().numpy()
    pick = np.concatenate([np.arange(200), np.arange(n - 200, n)])
    p = c[pick]
    want = rv_unit_columns(np.array([512.25]), 0.0, p[:, 0], p[:, 1], p[:, 2], p[:, 3])[:, 0]
    assert np.all(np.abs(got[pick] - want) <= 1e-9 / (1.0 - p[:, 1]) ** 2)
    assert np.all(np.isfinite(got))
