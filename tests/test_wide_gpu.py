"""GPU parity of the K-blocked 16-bit operands (g2_pack_blocked: fp16 counts
from u8 or u16 frames, signed digits) against the CPU oracle: N, S and D
bit-exact (int64), g2 equal to the oracle's FP64 value in float32.  The stacks
are small, so the size rule of the K-blocked operands is lifted."""
import numpy as np
import pytest

from oracle import g2_oracle as o
from test_dense_gpu import assert_exact

pytestmark = pytest.mark.gpu


def correlator(shape, T, qm, **over):
    from dynamix_gb300.correlator import MatMulCorrelator
    c = MatMulCorrelator(shape, T, qmask=qm)
    c.engine.NARROW_MIN_MACS = 0.0
    for k, v in over.items():
        setattr(c.engine, k, v)
    return c


def stack(T, shape, top, seed, dtype=np.uint16):
    rng = np.random.default_rng(seed)
    lam = top * rng.random((1,) + shape) ** 2 * (0.8 + 0.2 * rng.random((T, 1, 1)))
    fr = np.minimum(rng.poisson(lam), min(2 * top, np.iinfo(dtype).max)).astype(dtype)
    fr[rng.integers(T), rng.integers(shape[0]), rng.integers(shape[1])] = top
    return fr


@pytest.mark.parametrize("mode,dtype,top", [("fp16", np.uint8, 200), ("fp16", np.uint16, 300),
                                            ("bytes", np.uint16, 1024),     # 128 columns hold 2^24 and more
                                            ("bytes", np.uint16, 20000)])
@pytest.mark.parametrize("T", [1, 2, 31, 33, 127, 128, 129, 256, 257, 449, 700])
def test_ragged_frame_counts(built_lib, cuda_device, T, mode, dtype, top):
    import torch
    from dynamix_gb300.speckle import annular_qmask
    shape = (37, 61)
    fr = stack(T, shape, top, T, dtype)
    qm = annular_qmask(shape, 4, 1.0, 25.0)
    c = correlator(shape, T, qm)
    for _ in range(2):
        g = c.correlate(torch.from_numpy(fr).to(cuda_device))
        assert c.engine.last["mode"] == mode and c.engine.last["plan"] == "sampled"
        assert_exact(c, o.g2_exact(fr, qm), g)


@pytest.mark.parametrize("mode,dtype,top", [("fp16", np.uint8, 255), ("fp16", np.uint16, 300), (None, np.uint16, 900),
                                            ("bytes", np.uint16, 30000)])
@pytest.mark.parametrize("shape,rings", [((64, 96), None), ((5, 7), None), ((1, 2100), None), ((50, 83), 48),
                                         ((33, 130), "checker"), ((2, 4081), None)])
def test_layouts(built_lib, cuda_device, shape, rings, mode, dtype, top):
    """One bin of everything, chunk edges, narrow rings (mostly single pixels), interleaved bins."""
    import torch
    from dynamix_gb300.speckle import annular_qmask
    T = 200
    fr = stack(T, shape, top, 3, dtype)
    qm = None if rings is None else annular_qmask(shape, rings, 0.0, 40.0) if rings != "checker" else \
        (1 + np.arange(shape[0] * shape[1]) % 3).reshape(shape).astype(np.int32)
    c = correlator(shape, T, qm)
    g = c.correlate(torch.from_numpy(fr).to(cuda_device))
    assert c.engine.last["mode"] == (mode or c.engine.last["mode"]) and c.engine.last["plan"] == "sampled"
    assert_exact(c, o.g2_exact(fr, qm), g)


def test_every_digit(built_lib, cuda_device):
    """Every value of the low byte beside a few high bytes, the largest counts among them."""
    import torch
    shape, T = (4, 64), 256
    fr = np.zeros((T,) + shape, np.uint16)
    for p, hi in enumerate((0, 1, 127, 255)):
        fr[np.arange(T), p, (np.arange(T) * 7 + p) % 64] = np.arange(T) + 256 * hi
    c = correlator(shape, T, None)
    g = c.correlate(torch.from_numpy(fr).to(cuda_device))
    assert c.engine.last["mode"] == "bytes" and c.engine.last["plan"] == "sampled"
    assert_exact(c, o.g2_exact(fr, None), g)


def test_brighter_frames_than_sampled(built_lib, cuda_device):
    """A frame outside the sample that is far brighter than the K split allows
    is found by the Gram's own diagonal; counts above 2048 by the pack; both
    rerun, and the result is exact every time."""
    import torch
    shape, T = (64, 64), 300
    fr = stack(T, shape, 100, 1)
    x = torch.from_numpy(fr)
    c = correlator(shape, T, None)
    assert_exact(c, o.g2_exact(fr, None), c.correlate(x.to(cuda_device)))
    fr[7] = 1200                                          # 2^32.5 of energy, not among the 32 sampled frames
    assert 7 not in [(2 * k + 1) * T // 64 for k in range(32)]
    assert_exact(c, o.g2_exact(fr, None), c.correlate(x.to(cuda_device)))
    assert c.engine._wide_margin == 2 and c.engine.last["plan"] != "sampled"
    c = correlator(shape, T, None)
    fr[7] = 0
    fr[8, 3, 3] = 4000
    for _ in range(2):
        assert_exact(c, o.g2_exact(fr, None), c.correlate(x.to(cuda_device)))
        assert c.engine.last["mode"] == "bytes" and c.engine.last["plan"] == "sampled"


def test_host_frames_and_changing_stacks(built_lib, cuda_device):
    """Pinned host frames and device frames in turn, from single counts to
    bright and back, on one correlator."""
    import torch
    from dynamix_gb300.speckle import annular_qmask
    shape, T = (40, 100), 600
    qm = annular_qmask(shape, 5, 2.0, 30.0)
    c = correlator(shape, T, qm, NARROW_LOOK=3)
    for k, top in enumerate((8, 60, 60, 300, 300, 60, 60, 8, 8, 8, 5000, 5000)):
        fr = stack(T, shape, top, k)
        x = torch.from_numpy(fr)
        assert_exact(c, o.g2_exact(fr, qm), c.correlate(x.pin_memory() if k % 2 else x.to(cuda_device)))


@pytest.mark.parametrize("top", [500, 6000])
def test_deviation_and_two_time(built_lib, cuda_device, top):
    """calc_std and the two-time matrix of a K-blocked operand: the same as
    from a plain run, to their own rounding (float32 Gram entries; sums in
    another order)."""
    import torch
    from dynamix_gb300.correlator import MatMulCorrelator
    from dynamix_gb300.speckle import annular_qmask
    shape, T = (40, 44), 300
    qm = annular_qmask(shape, 3, 1.0, 20.0)
    x = torch.from_numpy(stack(T, shape, top, 5)).to(cuda_device)
    c, d = correlator(shape, T, qm), MatMulCorrelator(shape, T, qmask=qm)
    res, want = c.correlate(x, calc_std=True), d.correlate(x, calc_std=True)
    assert c.engine.last["plan"] == "sampled" and np.array_equal(res.res, want.res)
    assert np.allclose(res.dev, want.dev, rtol=1e-4, atol=1e-7, equal_nan=True)
    if top <= 2048:
        a, b = c.two_time(2), d.two_time(2)
        assert np.allclose(a, b, rtol=1e-6, atol=0, equal_nan=True)
