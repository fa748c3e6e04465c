"""GPU parity of the narrow operands of u8 stacks (csrc/g2_tail.cu: e2m1 and
e4m3 elements with residual lists; g2_gram_tc_e2m1) against the CPU oracle: N,
S and D bit-exact (int64), g2 equal to the oracle's FP64 value in float32.
The stacks are small, so the size rule of the narrow operands is lifted."""
import numpy as np
import pytest

from oracle import g2_oracle as o
from test_dense_gpu import assert_exact

pytestmark = pytest.mark.gpu


def correlator(shape, T, qm, **over):
    from dynamix_gb300.correlator import MatMulCorrelator
    c = MatMulCorrelator(shape, T, qmask=qm)
    c.engine.NARROW_MIN_MACS = 0.0
    share = over.pop("share", 5e-2)
    c.engine.NARROW_MAX = {3: share, 2: share}          # e2m1, e4m3
    for k, v in over.items():
        setattr(c.engine, k, v)
    return c


def stack(T, shape, mu, seed, peaks=0):
    from dynamix_gb300.speckle import speckle_numpy
    fr = speckle_numpy(T, shape, 0.97, mu, seed=seed)
    rng = np.random.default_rng(seed + 1)
    for _ in range(peaks):                       # single large counts, 255 among them
        fr[rng.integers(T), rng.integers(shape[0]), rng.integers(shape[1])] = rng.choice([5, 7, 8, 11, 15, 16, 17, 255])
    return fr


@pytest.mark.parametrize("mode,mu", [("e2m1", 0.6), ("e4m3", 2.0)])
@pytest.mark.parametrize("T", [1, 2, 31, 33, 127, 128, 223, 224, 225, 256, 257, 448, 449, 700, 1100])
def test_ragged_frame_counts(built_lib, cuda_device, T, mode, mu):
    import torch
    from dynamix_gb300.speckle import annular_qmask
    shape = (37, 61)
    fr = stack(T, shape, mu, T, peaks=6)
    qm = annular_qmask(shape, 4, 1.0, 25.0)
    c = correlator(shape, T, qm, _narrow_over={3} if mode == "e4m3" else set())
    g = c.correlate(torch.from_numpy(fr).to(cuda_device))
    assert c.engine.last["mode"] == mode and c.engine.last["residuals"] > 0
    assert_exact(c, o.g2_exact(fr, qm), g)


@pytest.mark.parametrize("mode", ["e2m1", "e4m3"])
@pytest.mark.parametrize("shape,rings", [((64, 96), None), ((5, 7), None), ((1, 2100), None), ((50, 83), 48),
                                         ((33, 130), "checker")])
def test_layouts(built_lib, cuda_device, shape, rings, mode):
    """One bin of everything, chunk edges, narrow rings (mostly single pixels), interleaved bins."""
    import torch
    from dynamix_gb300.speckle import annular_qmask
    T = 300
    fr = stack(T, shape, 0.4, 3, peaks=20)
    qm = None if rings is None else annular_qmask(shape, rings, 0.0, 40.0) if rings != "checker" else \
        (1 + np.arange(shape[0] * shape[1]) % 3).reshape(shape).astype(np.int32)
    c = correlator(shape, T, qm, _narrow_over={3} if mode == "e4m3" else set())
    g = c.correlate(torch.from_numpy(fr).to(cuda_device))
    assert c.engine.last["mode"] == mode
    assert_exact(c, o.g2_exact(fr, qm), g)


def test_every_count_value(built_lib, cuda_device):
    """Each u8 value once per pixel row, e2m1 and e4m3."""
    import torch
    shape, T = (8, 64), 256
    fr = np.zeros((T,) + shape, np.uint8)
    for p in range(8):
        fr[np.arange(T), p, (np.arange(T) * 7 + p) % 64] = np.arange(T)
    for over in (set(), {3}):
        c = correlator(shape, T, None, share=1.0, _narrow_over=over)
        g = c.correlate(torch.from_numpy(fr).to(cuda_device))
        assert c.engine.last["mode"] == ("e4m3" if over else "e2m1")
        assert_exact(c, o.g2_exact(fr, None), g)


def test_host_frames_and_mode_changes(built_lib, cuda_device):
    """Pinned host frames (cropped to the q-mask's columns) and device frames
    in turn, from dim to bright and back, on one correlator."""
    import torch
    from dynamix_gb300.speckle import annular_qmask
    shape, T = (40, 400), 600
    qm = annular_qmask(shape, 5, 2.0, 30.0, center=(20, 200))
    c = correlator(shape, T, qm, share=1e-3)
    seen = []
    for k, mu in enumerate((0.1, 1.5, 1.5, 30.0, 30.0, 0.1, 0.1)):
        fr = stack(T, shape, mu, k, peaks=3)
        x = torch.from_numpy(fr)
        g = c.correlate(x.pin_memory() if k % 2 else x.to(cuda_device))
        assert_exact(c, o.g2_exact(fr, qm), g)
        seen.append(c.engine.last["mode"])
    assert seen[0] == "e2m1" and "e4m3" in seen[1:3] and seen[4] == "fp16"


def test_overflowing_lists_take_a_wider_operand(built_lib, cuda_device):
    """A pixel that is bright in every frame overflows its sector's list."""
    import torch
    from dynamix_gb300.speckle import annular_qmask
    shape, T = (40, 44), 500
    qm = annular_qmask(shape, 3, 1.0, 20.0)
    fr = stack(T, shape, 0.1, 8)
    fr[:, 20, 10] = 9                                  # e2m1: a residual in every frame
    c = correlator(shape, T, qm, share=1e-3)            # 320 entries per list
    x = torch.from_numpy(fr).to(cuda_device)
    for _ in range(2):
        g = c.correlate(x)
        assert_exact(c, o.g2_exact(fr, qm), g)
    assert c.engine.last["mode"] == "e4m3" and 3 in c.engine._narrow_over


@pytest.mark.parametrize("mu", [0.2, 2.0])
def test_deviation_and_two_time_after_narrow_run(built_lib, cuda_device, mu):
    """calc_std and the two-time matrix expand a narrow operand back to the
    counts: the same values as from a plain run, to their own rounding (one
    float32 Gram entry per pair, exact; sums in another order)."""
    import torch
    from dynamix_gb300.correlator import MatMulCorrelator
    from dynamix_gb300.speckle import annular_qmask
    shape, T = (40, 44), 300
    qm = annular_qmask(shape, 3, 1.0, 20.0)
    fr = stack(T, shape, mu, 5, peaks=10)
    x = torch.from_numpy(fr).to(cuda_device)
    c = correlator(shape, T, qm)
    res = c.correlate(x, calc_std=True)
    assert "residuals" in c.engine.last
    d = MatMulCorrelator(shape, T, qmask=qm)
    want = d.correlate(x, calc_std=True)
    assert np.array_equal(res.res, want.res)
    assert np.allclose(res.dev, want.dev, rtol=1e-5, atol=1e-9, equal_nan=True)
    assert np.array_equal(c.two_time(2), d.two_time(2), equal_nan=True)


def test_fp32_accumulation_exact_e2m1(built_lib, cuda_device):
    """Gram entries of u u' just below 2^23 with odd low bits on kind::mxf4,
    large terms first and last along K, of both signs."""
    import torch
    n, m = ((1 << 23) - 8192) // 16, 900
    fr = np.full((4, 1, n + m), 3, np.uint8)          # u = 0
    fr[0, 0, :n], fr[0, 0, n:] = 7, 4                 # u = 4, 1
    fr[1, 0, :m], fr[1, 0, m:] = 2, 7                 # u = -1, 4
    fr[2, 0] = np.random.default_rng(1).integers(0, 8, n + m)
    fr[3, 0, 1::2] = 0                                # u = 0, -3
    u = fr.reshape(4, -1).astype(np.int64) - 3
    assert (1 << 22) < np.abs(u @ u.T).max() <= (1 << 23)
    c = correlator(fr.shape[1:], 4, None, exact_limit=1 << 25, share=1.0)
    c.correlate(torch.from_numpy(fr).to(cuda_device))
    assert c.engine.last["mode"] == "e2m1" and c.engine.last["n_grams"] == 1
    assert np.array_equal(c.numerator, o.g2_exact(fr, None)["numerator"])
