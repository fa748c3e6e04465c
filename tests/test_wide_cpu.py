"""CPU checks of the K-blocked 16-bit operands' layout and of their K split."""
import numpy as np
import pytest

from dynamix_gb300 import _lib
from dynamix_gb300.plan import MODE_BYTES, MODE_FP16, PAD, NarrowLayout
from dynamix_gb300.speckle import annular_qmask

CH = _lib.NARROW_CHUNK


def pack(L, frame):
    """The packed columns of one frame as the units say, and the writes per column."""
    out, writes = np.zeros(L.packed_cols, int), np.zeros(L.packed_cols, int)
    pad = np.concatenate([frame, np.zeros(CH, frame.dtype)]).astype(int)
    for c in range(L.n_chunks):
        for x, y, z, w in L.units.reshape(-1, 4)[L.unit_block_off[c] * 32:L.unit_block_off[c + 1] * 32].tolist():
            cls, dst = x >> 30, x & 0x3FFFFFFF
            if cls == 0:
                continue
            n = 8 if cls == 1 else 2
            if cls == 3:
                v = np.array([pad[c * CH + s] if s < CH else 0 for s in (y & 0xFFF, y >> 12 & 0xFFF)])
            else:
                assert (y & 0xFFFF) <= CH - n
                v = pad[c * CH + (y & 0xFFFF):][:n]
            planes = [(0, v)] if not L.split else [(0, (v >> 8) + (v >> 7 & 1)), (w // 2, ((v & 255) ^ 128) - 128)]
            for off, e in planes:
                out[dst * n + off:dst * n + off + n] = e
                writes[dst * n + off:dst * n + off + n] += 1
    return out, writes


@pytest.mark.parametrize("mode", [MODE_FP16, MODE_BYTES])
@pytest.mark.parametrize("q,bins", [
    (annular_qmask((37, 61), 4, 2, 25), 4), (annular_qmask((90, 95), 48, 0, 45), 48), (np.ones((5, 7), np.int32), 1),
    (np.ones((1, CH + 1), np.int32), 1), (np.zeros((9, 11), np.int32), 2),
    ((1 + np.arange(4000) % 3).reshape(40, 100).astype(np.int32), 3)])
def test_layout(q, bins, mode):
    L = NarrowLayout(q, bins, mode)
    frame = np.random.default_rng(0).integers(0, 65536, q.size).astype(np.uint16)
    out, writes = pack(L, frame)
    assert writes.max(initial=0) <= 1 and L.packed_bytes_per_frame == 2 * L.packed_cols
    assert np.array_equal(L.ones_row_values(), (L.col_src >= 0).astype(np.uint16))
    S, N = np.zeros(bins, np.int64), np.zeros(bins, np.int64)
    for b, a, c, k, shift in L.grams():
        assert k % PAD == 0
        N[b] += int(out[a:a + k] @ out[c:c + k]) << shift
        if a == c:
            S[b] += int(out[a:a + k].sum()) << (shift // 2)
    f = frame.astype(np.int64)
    assert np.array_equal(S, [f[q.ravel() == b + 1].sum() for b in range(bins)])
    assert np.array_equal(N, [(f[q.ravel() == b + 1] ** 2).sum() for b in range(bins)])


@pytest.mark.parametrize("mode", [MODE_FP16, MODE_BYTES])
def test_split_covers_every_column_once_below_the_limit(mode):
    L = NarrowLayout(annular_qmask((90, 95), 5, 0, 45), 5, mode)
    e = np.random.default_rng(1).integers(0, 1000, (7, 1 + L.split, L.unit_col.size))
    cut = L.sampled_grams(e, 4000.0)
    assert L.split_peak(e, cut) <= 4000.0 and L.sampled_grams(e, 500.0) is None
    for g in L.grams():
        mine = sorted((k0, kl) for (b, a, c, k0, kl, s) in cut if (b, a, c, s) == (g[0], g[1], g[2], g[4]))
        assert mine[0][0] == 0 and sum(kl for _, kl in mine) == g[3]
        assert all(p + n == q for (p, n), (q, _) in zip(mine[:-1], mine[1:]))
