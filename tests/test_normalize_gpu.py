"""GPU parity of the one-launch normalisation (g2_normalize): D and the largest
S bit-exact in int64, g2 equal to float64 on the host, on a dirty denominator buffer."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 3, 80])
@pytest.mark.parametrize("T", [1, 2, 127, 128, 129, 1023, 1024, 1025, 2050, 5000])
@pytest.mark.parametrize("top", [1, 3000, 1 << 24, 1 << 25])
def test_normalize(built_lib, cuda_device, T, rows, top):
    import torch
    from dynamix_gb300 import _lib
    rng = np.random.default_rng(T + rows)
    S = rng.integers(0, top + 1, (rows, T))
    if T > 2 and top > 1 << 24:
        S[0, T // 2] = (1 << 33) // T                        # wider than the other windows
    N = rng.integers(0, 1 << 40, (rows, T))
    scale = rng.random(rows) + 0.5
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda_device)
    n, s, sc = d(N), d(S), d(scale)
    length = rows * T + (rows * -(-T // 1024) + 1) // 2
    den = torch.full((length,), -7, dtype=torch.int64, device=cuda_device)
    g32 = torch.empty((rows, T), dtype=torch.float32, device=cuda_device)
    g64 = torch.empty((rows, T), dtype=torch.float64, device=cuda_device)
    most = torch.zeros(1, dtype=torch.int64, device=cuda_device)
    p = lambda t: C.c_void_p(t.data_ptr())
    st = C.c_void_p(torch.cuda.current_stream(cuda_device).cuda_stream)
    for _ in range(2):
        _lib.check(built_lib.g2_normalize(p(n), p(s), p(sc), rows, T, p(den), length, p(g32), p(g64), p(most), st),
                   "g2_normalize")
    D = np.stack([np.array([int(np.dot(x[:T - t].astype(object), x[t:].astype(object))) if T <= 129 else 0
                            for t in range(T)], dtype=np.int64) for x in S]) if T <= 129 else None
    got = den[:rows * T].view(rows, T).cpu().numpy()
    if D is None:                                             # the lags at the block edges
        taus = sorted({0, 1, 2, T - 1, T // 2} | {t for t in (1022, 1023, 1024, 1025, 2047, 2048) if t < T})
        D = np.stack([[int(np.dot(x[:T - t].astype(object), x[t:].astype(object))) for t in taus] for x in S])
        assert np.array_equal(got[:, taus], D.astype(np.int64))
    else:
        assert np.array_equal(got, D)
    assert int(most.item()) == S.max()
    with np.errstate(divide="ignore", invalid="ignore"):
        want = scale[:, None] * N.astype(np.float64) / got.astype(np.float64)
    assert np.array_equal(g64.cpu().numpy(), want, equal_nan=True)
    assert np.array_equal(g32.cpu().numpy(), want.astype(np.float32), equal_nan=True)


def test_normalize_refuses_a_short_buffer(built_lib, cuda_device):
    import torch
    z = torch.zeros(64, dtype=torch.int64, device=cuda_device)
    p = C.c_void_p(z.data_ptr())
    assert built_lib.g2_normalize(p, p, p, 1, 32, p, 32, p, None, None, None) != 0
