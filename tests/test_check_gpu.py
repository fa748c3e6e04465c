"""GPU checks of event lists and CSR stacks that are used where they are
(csrc/g2_check.cu): what was refused is refused with the same exception, and
arrays at any alignment give the oracle's exact sums."""
import numpy as np
import pytest

from oracle import g2_oracle as o
from test_dense_gpu import assert_exact

pytestmark = pytest.mark.gpu


def frames(T, shape, seed, dtype=np.uint8, top=4):
    rng = np.random.default_rng(seed)
    return (rng.integers(1, top + 1, (T,) + shape) * (rng.random((T,) + shape) < 0.05)).astype(dtype)


def event_lists(fr):
    flat = fr.reshape(fr.shape[0], -1).T
    pix, t = np.nonzero(flat)
    return t.astype(np.int32), flat[pix, t], np.concatenate([[0], np.cumsum((flat > 0).sum(1))])


def csr(fr):
    T, H, W = fr.shape
    t, r, c = np.nonzero(fr)
    per = np.zeros((T, H), np.int64)
    np.add.at(per, (t, r), 1)
    ip = np.concatenate([np.zeros((T, 1), np.int64), np.cumsum(per, 1)], 1).astype(np.int32).ravel()
    return fr[t, r, c], c.astype(np.int32), ip, np.concatenate([[0], np.cumsum(per.sum(1))])


def shifted(a, dev, k):
    """The array on the device, ``k`` elements off an aligned start and with unused elements behind."""
    import torch
    pad = np.concatenate([np.zeros(k, a.dtype), a, np.full(3, 1, a.dtype)])
    return torch.from_numpy(pad).to(dev)[k:]


@pytest.mark.parametrize("k", [0, 1, 3])
@pytest.mark.parametrize("dtype,top", [(np.uint8, 255), (np.uint16, 255), (np.uint16, 3000)])
@pytest.mark.parametrize("ot", [np.int32, np.int64])
def test_events_in_place(built_lib, cuda_device, k, dtype, top, ot):
    from dynamix_gb300.correlator import EventCorrelator
    shape, T = (9, 31), 260
    fr = frames(T, shape, 1, dtype, top)
    t, v, off = event_lists(fr)
    c = EventCorrelator(shape, T, T, qmask=None)
    g = c.correlate(shifted(t, cuda_device, k), shifted(v, cuda_device, k), shifted(off.astype(ot), cuda_device, k)[:off.size])
    assert c.engine.last["max_count"] == v.max() and c.engine.last["n_events"] == v.size
    assert_exact(c, o.g2_exact(fr, None), g)


def test_bad_events_are_refused(built_lib, cuda_device):
    import torch
    from dynamix_gb300.correlator import EventCorrelator
    shape, T = (9, 31), 260
    t, v, off = event_lists(frames(T, shape, 2))
    c = EventCorrelator(shape, T, T, qmask=None)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda_device)

    def refused(t, v, off):
        with pytest.raises(ValueError):
            c.correlate_device(d(t), d(v), d(off))

    for at, val in ((0, -1), (t.size - 1, T), (t.size // 2, 2 ** 31 - 1)):
        bad = t.copy()
        bad[at] = val
        refused(bad, v, off)
    for at, val in ((0, 1), (5, off[6] + 1), (off.size - 1, off[-2] - 1), (off.size - 1, t.size + 1), (3, -4)):
        bad = off.copy()
        bad[at] = val
        refused(t, v, bad)
    none = np.zeros_like(off)
    assert np.isnan(c.correlate(d(t), d(v), d(none))).all() and c.engine.last["n_events"] == 0
    bad = t.copy()
    bad[-1] = T                                             # behind the last offset: not an event
    less = np.minimum(off, t.size - 1)
    c.correlate(d(bad), d(v), d(less))


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("ot", [np.int32, np.int64])
def test_csr_in_place(built_lib, cuda_device, dtype, ot):
    import torch
    from dynamix_gb300.correlator import SparseCorrelator
    from dynamix_gb300.engine import DeviceError
    shape, T = (11, 45), 1100
    fr = frames(T, shape, 3, dtype, 200)
    v, col, ip, off = csr(fr)
    qm = (1 + np.arange(fr[0].size) % 4).reshape(shape).astype(np.int32)
    c = SparseCorrelator(shape, T, qmask=qm)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda_device)
    good = (d(v), d(col), d(ip), d(off.astype(ot)))
    ref = o.g2_exact(fr, qm)
    assert_exact(c, ref, c.correlate(*good))
    for k in (1, 3):
        assert_exact(c, ref, c.correlate(shifted(v, cuda_device, k)[:v.size], shifted(col, cuda_device, k)[:v.size],
                                         good[2], good[3]))
    for at, val in ((0, -1), (v.size - 1, shape[1]), (v.size // 2, 2 ** 31 - 1)):
        bad = col.copy()
        bad[at] = val
        with pytest.raises(ValueError):
            c.correlate_device(good[0], d(bad), good[2], good[3])
    tail = np.concatenate([col, np.array([shape[1]], np.int32)])   # a bad column that no row points to
    with pytest.raises(ValueError):
        c.correlate_device(d(np.append(v, v[:1])), d(tail), good[2], good[3])
    swap = col.copy()
    f = int(np.flatnonzero(np.diff(ip.reshape(T, -1)[7]) >= 2)[0])
    e = int(off[7] + ip.reshape(T, -1)[7, f])
    swap[[e, e + 1]] = swap[[e + 1, e]]
    with pytest.raises(DeviceError):
        c.correlate(good[0], d(swap), good[2], good[3])
    far = off.astype(np.int64).copy()
    far[-1] = 2 ** 31
    with pytest.raises((DeviceError, ValueError)):
        c.correlate(good[0], good[1], good[2], d(far))
    assert_exact(c, ref, c.correlate(*good))
