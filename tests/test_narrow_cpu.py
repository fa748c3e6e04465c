"""CPU checks of the narrow operands' layout and of the K cut of short launches."""
import numpy as np
import pytest

from dynamix_gb300 import _lib
from dynamix_gb300.plan import (MODE_E2M1, MODE_E4M3, NarrowLayout, balance_items, chunk_grams, e2m1_segment_bound, gram_items, item_costs,
                                split_items)
from dynamix_gb300.speckle import annular_qmask

CH = _lib.NARROW_CHUNK


def pack(L, frame):
    """The packed columns of one frame as the units say, and the writes per byte."""
    e2m1 = L.mode == MODE_E2M1
    out = np.full(L.packed_cols, -1, int)
    writes = np.zeros(L.packed_bytes_per_frame, int)
    pad = np.concatenate([frame, np.zeros(CH, np.uint8)])
    for c in range(L.n_chunks):
        for x, y, z, w in L.units.reshape(-1, 4)[L.unit_block_off[c] * 32:L.unit_block_off[c + 1] * 32].tolist():
            cls, dst, base = x >> 30, x & 0x3FFFFFFF, c * CH
            if cls == 0:
                continue
            n = 16 if cls == 1 else 4
            if cls == 3:
                s = [((y | z << 32 | w << 64) >> 12 * k) & 0xFFF for k in range(8)]
                v = np.array([int(pad[base + k]) if k < CH else -1 for k in s])
                a, b = v[:4], v[4:]
            else:
                assert (y & 0xFFFF) <= CH - n and (y >> 16) <= CH - n
                a, b = pad[base + (y & 0xFFFF):][:n].astype(int), pad[base + (y >> 16):][:n].astype(int)
            if e2m1:
                a, b = a.reshape(-1, 4), b.reshape(-1, 4)        # columns a0 a2 b0 b2 a1 a3 b1 b3 of every word
                v = np.stack([a[:, 0], a[:, 2], b[:, 0], b[:, 2], a[:, 1], a[:, 3], b[:, 1], b[:, 3]], 1).ravel()
            else:
                v = a
            out[dst * v.size:dst * v.size + v.size] = v
            writes[dst * n:dst * n + n] += 1
    return out, writes


@pytest.mark.parametrize("mode", [MODE_E2M1, MODE_E4M3])
@pytest.mark.parametrize("q,bins", [
    (annular_qmask((37, 61), 4, 2, 25), 4), (annular_qmask((130, 127), 8, 0, 64), 8),
    (annular_qmask((90, 95), 48, 0, 45), 48), (np.ones((5, 7), np.int32), 1), (np.ones((1, CH + 1), np.int32), 1),
    (np.zeros((9, 11), np.int32), 2), ((1 + np.arange(4000) % 3).reshape(40, 100).astype(np.int32), 3),
    (np.where(np.arange(9000) == CH, 2, 0).reshape(90, 100).astype(np.int32), 3)])
def test_narrow_layout(q, bins, mode):
    L = NarrowLayout(q, bins, mode)
    frame = np.random.default_rng(0).integers(0, 8, q.size).astype(np.uint8)
    out, writes = pack(L, frame)
    assert writes.max(initial=0) <= 1
    assert np.array_equal(out, np.where(L.col_src >= 0, frame[L.col_src].astype(int), -1))
    assert L.packed_bytes_per_frame % 128 == 0 and L.sector_bin.size * 64 == L.packed_cols
    for b in range(bins):                                     # every bin holds its pixels once, bin padding nothing
        seg = L.col_src[L.bin_off[b]:L.bin_off[b] + L.kpad[b]]
        assert np.array_equal(np.sort(seg[seg >= 0]), np.flatnonzero(q.ravel() == b + 1))
        assert np.all(L.sector_bin[L.bin_off[b] // 64:(L.bin_off[b] + L.kpad[b]) // 64] == b)
    ones = L.ones_row_values()
    if mode == MODE_E2M1:
        ones = np.stack([ones & 15, ones >> 4], 1).ravel()
    assert np.array_equal(ones, (L.col_src >= 0).astype(np.uint8))
    for c in range(L.n_chunks):                               # spans cover the chunk's binned pixels
        p = np.flatnonzero(q.ravel()[c * CH:(c + 1) * CH] > 0)
        lo, hi = int(L.chunk_span[c]) & 0xFFFF, int(L.chunk_span[c]) >> 16
        assert (p.size == 0 and L.unit_block_off[c] == L.unit_block_off[c + 1]) or (lo <= p[0] and p[-1] < hi <= CH)


@pytest.mark.parametrize("T,workers", [(100, 76), (1777, 76), (600, 3), (600, 1)])
def test_split_items_cover_every_column_once(T, workers):
    L = NarrowLayout(annular_qmask((200, 210), 5, 3, 90), 5)
    items = gram_items(T, chunk_grams(L, e2m1_segment_bound(L)), kind="pair4", s_base=0)
    parts = split_items(items, workers, 256, "pair4")
    whole = {}
    for it in items:
        whole[(int(it["i0"]), int(it["j0"]), int(it["out_off"]))] = (int(it["a_k0"]), int(it["k_len"]))
    got = {}
    for it in parts:
        assert it["k_len"] > 0 and it["k_len"] % 256 == 0 and it["a_k0"] == it["b_k0"] and it["a_k0"] % 256 == 0
        got.setdefault((int(it["i0"]), int(it["j0"]), int(it["out_off"])), []).append((int(it["a_k0"]), int(it["k_len"])))
    assert got.keys() == whole.keys()
    for k, pieces in got.items():
        pieces.sort()
        assert pieces[0][0] == whole[k][0] and sum(n for _, n in pieces) == whole[k][1]
        assert all(a + n == b for (a, n), (b, _) in zip(pieces, pieces[1:]))
    if workers == 76 and T == 100:                            # 5 bins, one tile each: the GPU is filled
        assert parts.size > items.size
    out = balance_items(parts, workers, 256, "pair4")
    assert (out["job"] >= 0).sum() == parts.size and item_costs(parts, 256, "pair4").min() > 0
