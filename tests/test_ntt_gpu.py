"""G3 and G4 by number-theoretic transforms (g2_normalize_ntt): D equal to the
int64 autocorrelation and g2 to g2_finalize's, from one frame to several blocks
of 2,048, for sums up to the largest whose D fits int64."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 2, 3, 4, 5, 31, 64, 257, 512, 1000, 1024, 1025, 2047, 2048, 2049, 4096, 4097, 5000,
                               6143, 10007])
@pytest.mark.parametrize("rows", [1, 5])
def test_matches_direct(built_lib, cuda_device, T, rows):
    import torch
    from dynamix_gb300.engine import ntt_roots
    rng = np.random.default_rng(T + rows)
    S = np.zeros((rows, T), np.int64)
    S[0] = rng.integers(0, int((2.0 ** 63 / T) ** 0.5), T)                # D up to 2^63
    for r in range(1, rows):
        S[r] = rng.integers(0, 10 ** r, T)
    S[-1, : T // 2] = 0
    N = rng.integers(0, 2 ** 50, (rows, T))
    d = lambda a: torch.from_numpy(a).to(cuda_device)
    p = lambda t: C.c_void_p(t.data_ptr())
    s, n, scale = d(S), d(N), d(rng.random(rows) * 1000 + 1)
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    out = []
    for ntt in (False, True):
        D = torch.full((rows, T), -1, dtype=torch.int64, device=cuda_device)
        f = torch.full((rows, T), -1.0, dtype=torch.float32, device=cuda_device)
        g = torch.full((rows, T), -1.0, dtype=torch.float64, device=cuda_device)
        if ntt:
            k = built_lib.g2_ntt_scratch(rows, T)
            buf = torch.empty(max(k, 1), dtype=torch.int64, device=cuda_device)
            assert built_lib.g2_normalize_ntt(p(n), p(s), p(scale), rows, T, p(ntt_roots(cuda_device)), p(buf), k, p(D),
                                              p(f), p(g), st) == 0
            assert built_lib.g2_normalize_ntt(p(n), p(s), p(scale), rows, T, p(ntt_roots(cuda_device)), p(buf), k, p(D),
                                              None, None, st) == 0
            if k:
                assert built_lib.g2_normalize_ntt(p(n), p(s), p(scale), rows, T, p(ntt_roots(cuda_device)), p(buf),
                                                  k - 1, p(D), p(f), p(g), st) != 0
        else:
            assert built_lib.g2_denominator(p(s), rows, T, p(D), st) == 0
            assert built_lib.g2_finalize(p(n), p(D), p(scale), rows, T, p(f), p(g), st) == 0
        out.append([x.cpu().numpy() for x in (D, f, g)])
    for a, b in zip(*out):
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f")


@pytest.mark.parametrize("T", [1, 127, 128, 129, 1000, 1024, 1025, 2300])
@pytest.mark.parametrize("rows", [1, 9, 400])
def test_short_windows_of_the_direct_kernel(built_lib, cuda_device, T, rows):
    """g2_denominator's 128-frame windows (launches of few blocks) and 1024-frame ones against numpy."""
    import torch
    S = np.random.default_rng(T).integers(0, 70000, (rows, T))
    s = torch.from_numpy(S).to(cuda_device)
    D = torch.full((rows, T), -1, dtype=torch.int64, device=cuda_device)
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert built_lib.g2_denominator(C.c_void_p(s.data_ptr()), rows, T, C.c_void_p(D.data_ptr()), st) == 0
    got = D.cpu().numpy()
    for r in {0, rows // 2, rows - 1}:
        assert np.array_equal(got[r], np.correlate(S[r], S[r], "full")[T - 1:])
