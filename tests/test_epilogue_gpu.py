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


@pytest.mark.parametrize("dtype,top", [(np.uint8, 6), (np.uint8, 40), (np.uint16, 300)])
def test_two_time_of_a_bin_of_a_blocked_operand(built_lib, cuda_device, dtype, top):
    """Only the bin's columns of a K-blocked operand are copied to rows: bins at
    the start, in the middle and at the end, an empty one, residuals in others."""
    import torch
    from dynamix_gb300.correlator import MatMulCorrelator
    rng = np.random.default_rng(top)
    T, shape = 270, (30, 40)
    fr = rng.poisson(top / 3.0 * rng.random((1,) + shape), (T,) + shape).clip(0, top).astype(dtype)
    fr[5, 3, 7], fr[9, 20, 30] = top, min(3 * top, 255)
    qm = np.repeat([1, 2, 0, 4], 300).reshape(shape).astype(np.int32)
    c = MatMulCorrelator(shape, T, qmask=qm)
    c.engine.NARROW_MIN_MACS = 0.0
    c.engine.NARROW_MAX = {3: 1e-2, 2: 1e-2}
    c.correlate(torch.from_numpy(fr).to(cuda_device))
    assert c.engine._packed_layout[0]
    for q in (1, 2, c.n_bins):
        if not np.any(qm == q):
            continue
        got, want = c.two_time(q), o.ttcf_exact(fr, qm, q)
        ok = np.isfinite(want)
        assert np.array_equal(np.isfinite(got), ok)
        assert np.all(np.abs(got[ok] - want[ok]) <= 5e-6 * np.abs(want[ok]) + 1e-30)
