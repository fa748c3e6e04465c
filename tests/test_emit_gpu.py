"""The event lists straight from the frames (g2_compress_emit) against the host
compressor: steps that fit the shared buffer and steps that do not, ragged
frame and pixel counts (rows at every alignment), all element types."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.uint8, np.int8, np.uint16, np.int16])
@pytest.mark.parametrize("shape", [(1, 1), (1, 3), (4, 33), (16, 16), (7, 73), (13, 79)])
@pytest.mark.parametrize("T", [1, 31, 33, 511, 513, 1024, 1025, 2300])
@pytest.mark.parametrize("fill", [0.09, 1.0])
def test_emit(built_lib, cuda_device, dtype, shape, T, fill):
    import torch
    from dynamix_gb300.correlator import FramesCompressor
    rng = np.random.default_rng(T + shape[1])
    info = np.iinfo(dtype)
    fr = rng.integers(1, info.max, (T,) + shape, endpoint=True).astype(dtype)
    fr[rng.random(fr.shape) >= fill] = 0
    if info.min < 0:
        fr[rng.random(fr.shape) < 0.05] = info.min            # negative values are no events
    want = FramesCompressor.compress_all_stack(fr)
    got = FramesCompressor.compress_all_stack(torch.from_numpy(fr).to(cuda_device))
    for w, g in zip(want, got):
        assert np.array_equal(w, g.cpu().numpy().astype(w.dtype))
    assert got[0].cpu().numpy().dtype == dtype and got[1].dtype == torch.int32
