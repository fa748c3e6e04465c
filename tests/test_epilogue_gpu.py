"""Deviation and two-time epilogues of the Gram at the edges of their tiles
(128 rows, 256 columns, chunks of 32) against the float64 oracle, with the
tolerances of the larger cases: 1e-4 relative for the deviation, 5e-6 for the
two-time ratios (float32 products, quotients and sums)."""
import numpy as np
import pytest

from oracle import g2_oracle as o

pytestmark = pytest.mark.gpu


def stack(T, empty, seed=3):
    from dynamix_gb300.speckle import speckle_numpy
    fr = speckle_numpy(T, (20, 26), 0.97, 0.8, seed=seed)
    if empty:
        fr[min(3, T - 1)::9] = 0
    return fr, (1 + (np.arange(20 * 26) % 3 == 0) + (np.arange(20 * 26) > 300)).reshape(20, 26).astype(np.int32)


@pytest.mark.parametrize("empty", [False, True])
@pytest.mark.parametrize("T", [1, 2, 31, 32, 33, 127, 128, 129, 159, 160, 161, 255, 256, 257, 287, 385, 700])
def test_deviation_tile_edges(built_lib, cuda_device, T, empty):
    import torch
    from dynamix_gb300.correlator import MatMulCorrelator
    fr, qm = stack(T, empty)
    c = MatMulCorrelator(fr.shape[1:], T, qmask=qm)
    c.correlate(torch.from_numpy(fr).to(cuda_device), calc_std=True)
    want, got = o.dense_std_exact(fr, qm), c.engine.dev_f64[: c.n_bins].cpu().numpy()
    ok = np.isfinite(want)
    assert np.array_equal(np.isfinite(got), ok)
    assert np.all(np.abs(got[ok] - want[ok]) <= 1e-4 * np.abs(want[ok]) + 1e-9)


@pytest.mark.parametrize("empty", [False, True])
@pytest.mark.parametrize("T", [7, 33, 130, 256, 259, 260, 385, 387, 644])
def test_two_time_tile_edges(built_lib, cuda_device, T, empty):
    import torch
    from dynamix_gb300.correlator import MatMulCorrelator
    fr, qm = stack(T, empty, 5)
    c = MatMulCorrelator(fr.shape[1:], T, qmask=qm)
    c.correlate(torch.from_numpy(fr).to(cuda_device))
    for q in (1, 3):
        got, want = c.two_time(q), o.ttcf_exact(fr, qm, q)
        assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
        ok = np.isfinite(want)
        assert np.all(np.abs(got[ok] - want[ok]) <= 5e-6 * np.abs(want[ok]) + 1e-30)
