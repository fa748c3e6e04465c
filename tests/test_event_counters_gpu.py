"""GPU parity of the event pair sums round their block edges and with uint32
counters that wrap: N and S bit-exact (int64) against the CPU oracle on the
dense frames the lists hold."""
import numpy as np
import pytest

from oracle import g2_oracle as o
from test_dense_gpu import assert_exact

pytestmark = pytest.mark.gpu


def lists(fr):
    """(frames, counts, offsets) of the pixels' events, frame order within a pixel."""
    flat = fr.reshape(fr.shape[0], -1).T
    pix, t = np.nonzero(flat)
    return t.astype(np.int32), flat[pix, t], np.concatenate([[0], np.cumsum((flat > 0).sum(1))]).astype(np.uint32)


@pytest.mark.parametrize("T,events", [(301, (0, 1, 7, 8, 9, 16, 17, 60)), (400, (127, 128, 129, 136, 255, 256, 257)),
                                      (999, (384, 500, 640)), (64, (24,) * 5), (64, (23,) * 5)])
@pytest.mark.parametrize("top", [1, 200, 30000])
def test_events_per_pixel(built_lib, cuda_device, T, events, top):
    """Lists of every length round the row and block edges, odd frame counts,
    counts whose sums wrap a counter (30000: within five adds), events in random order."""
    import torch
    from dynamix_gb300.correlator import EventCorrelator
    rng = np.random.default_rng(T + top)
    shape = (6, 60)
    fr = np.zeros((T, shape[0] * shape[1]), np.uint16 if top > 255 else np.uint8)
    for p in range(fr.shape[1]):
        n = min(T, events[p % len(events)])
        fr[rng.permutation(T)[:n], p] = rng.integers(1, top + 1, n)
    fr = fr.reshape((T,) + shape)
    qm = (1 + np.arange(fr[0].size) % 3).reshape(shape).astype(np.int32)
    qm[0, :7] = 0
    t, v, off = lists(fr)
    for p in range(0, off.size - 1, 2):
        s = slice(off[p], off[p + 1])
        k = rng.permutation(off[p + 1] - off[p])
        t[s], v[s] = t[s][k], v[s][k]
    c = EventCorrelator(shape, T, int(np.diff(off).max()), qmask=qm)
    d = lambda a: torch.from_numpy(a).to(cuda_device)
    g = c.correlate(d(t), d(v), d(off.astype(np.int32)))
    assert_exact(c, o.g2_exact(fr, qm), g)
