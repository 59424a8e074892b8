"""The plain GEMM's k segments: their plan on the CPU, their results on the GPU."""
import ctypes as C

import numpy as np
import pytest

import ca3dmm_b200 as cb


class Seg(C.Structure):
    _fields_ = [(n, C.c_int) for n in ("tm", "tn", "kt0", "kt1", "part", "nparts", "slot0", "counter")]


def segments(m, n, k, tile_n):
    L = cb.lib()
    mx = L.ca3dmm_dgemm_segments_max(m, n, k)
    if mx == 0:
        return None
    segs, order, begin = (Seg * mx)(), (C.c_int * mx)(), (C.c_int * 149)()
    ns, grid, nc = C.c_int(), C.c_int(), C.c_int()
    assert L.ca3dmm_dgemm_segments(m, n, k, tile_n, segs, order, begin, C.byref(ns), C.byref(grid),
                                   C.byref(nc)) == 0
    assert ns.value <= mx
    L.ca3dmm_dgemm_segments_ws_bytes.restype = C.c_size_t
    return (segs[:ns.value], list(order[:ns.value]), list(begin[:grid.value + 1]), grid.value,
            nc.value, L.ca3dmm_dgemm_segments_ws_bytes(m, n, k))


SHAPES = [(1, 1, 1), (200, 150, 300), (128, 128, 100000), (129, 64, 17), (1000, 1000, 1000),
          (1501, 2003, 3001), (2048, 2048, 2048), (2048, 2048, 64), (3200, 3100, 1500),
          (5000, 640, 33), (128 * 148, 128, 512), (4000, 5000, 1200), (16384, 130, 500)]


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_segments_cover_every_block_once(m, n, k):
    got = {t: segments(m, n, k, t) for t in (128, 64)}
    if got[128] is None:
        assert got[64] is None
        return
    cuts = {}
    for tile_n, (segs, order, begin, grid, nc, ws) in got.items():
        assert 1 <= grid <= 148 and nc <= 2 * 148
        assert sorted(order) == list(range(len(segs)))
        assert begin[0] == 0 and begin[-1] == len(segs) and begin == sorted(begin)
        K = -(-k // 16)
        tiles, slots, counters = {}, set(), set()
        for i, s in enumerate(segs):
            tiles.setdefault((s.tm, s.tn), []).append(s)
            assert i == 0 or segs[i - 1].tm // 8 <= s.tm // 8           # bands of 8 tile rows
        assert set(tiles) == {(i, j) for i in range(-(-m // 128)) for j in range(-(-n // tile_n))}
        for key, l in tiles.items():
            assert [s.part for s in l] == list(range(len(l))) and all(s.nparts == len(l) for s in l)
            assert l[0].kt0 == 0 and l[-1].kt1 == K
            assert all(a.kt1 == b.kt0 for a, b in zip(l, l[1:])) and all(s.kt0 < s.kt1 for s in l)
            if len(l) > 1:
                assert all(s.slot0 == l[0].slot0 and s.counter == l[0].counter for s in l)
                mine = set(range(l[0].slot0, l[0].slot0 + len(l)))
                assert not mine & slots and l[0].counter not in counters
                slots |= mine
                counters.add(l[0].counter)
                assert l[0].counter < nc
        if slots:
            assert (max(slots) + 1) * 128 * tile_n * 8 <= ws
        # the cuts of a 128-column tile, whatever the width
        cuts[tile_n] = {(tm, tn * tile_n // 128): [s.kt0 for s in l] for (tm, tn), l in tiles.items()}
        # shares are equal in 128-column blocks (a 64-column half past n costs nothing)
        if tile_n == 128 and len(segs) > grid and any(s.nparts > 1 for s in segs):
            load = [sum(segs[i].kt1 - segs[i].kt0 for i in order[begin[b]:begin[b + 1]])
                    for b in range(grid)]
            share = sum(load) / grid
            assert max(load) <= share * 1.15 + 3, (max(load), share)
    assert cuts[64] == cuts[128]


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,ta,tb,p", [
    (1, 1, 1, 0, 0, 1), (128, 128, 5000, 0, 0, 1), (129, 131, 257, 1, 1, 4), (200, 150, 300, 0, 0, 4),
    (1000, 999, 1000, 1, 0, 1), (640, 700, 4097, 0, 1, 6), (1501, 2003, 301, 1, 1, 6),
    (2500, 1300, 777, 0, 0, 8), (3200, 3100, 500, 0, 0, 3),
])
def test_segments_against_double_double(cuda, monkeypatch, m, n, k, ta, tb, p):
    """Within k u |A||B| of the double-double truth (the bound of one chain of k
    additions), the same bits from two execs, and at most the error of the kp
    slabs they replace plus a margin of 3 u."""
    from oracle import oracle as orc
    from tests._util import dev_zeros, from_dev, to_dev
    A = orc.gen_signed_exp(5, *((k, m) if ta else (m, k)))
    B = orc.gen_signed_exp(6, *((n, k) if tb else (k, n)))
    dA, lda = to_dev(A)
    dB, ldb = to_dev(B)
    ii, jj = orc.sample_indices(m, n, nrand=2000, nlines=2)
    hi, lo, ab = orc.dd_entries(A, B, ta, tb, k, ii, jj)
    err = {}
    for merge in ("1", "0"):
        monkeypatch.setenv("CA3DMM_PLAIN_MERGE_SLABS", merge)
        e = cb.Ca3dmmEngine(m, n, k, ta, tb, p=p)
        outs = []
        for _ in range(2):
            dC = dev_zeros(m * n)
            assert e.ok and e.exec(dA, lda, dB, ldb, dC, m) == 0
            outs.append(from_dev(dC, m, n))
        e.free()
        assert np.array_equal(outs[0], outs[1])
        d = np.abs((outs[0][ii, jj] - hi) - lo)
        assert np.all(d <= k * 2.0 ** -53 * ab)
        err[merge] = np.sqrt(np.mean((d / ab) ** 2))
    assert err["1"] <= 1.1 * err["0"] + 3 * 2.0 ** -53 / np.sqrt(k), err


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,p", [(300, 200, 400, 1), (1000, 900, 800, 4)])
def test_buffer_sized_in_split_mode_serves_plain(cuda, monkeypatch, m, n, k, p):
    """A caller's work buffer of the size asked for in a split-precision mode
    holds the plain mode's layout."""
    import torch
    from tests._util import dev_zeros, from_dev, to_dev
    A, B = np.random.default_rng(1).standard_normal((m, k)), np.random.default_rng(2).standard_normal((k, n))
    dA, lda = to_dev(A)
    dB, ldb = to_dev(B)
    outs = []
    for mode in ("0", "1", "2"):
        monkeypatch.setenv("CA3DMM_GEMM_MODE", mode)
        e = cb.Ca3dmmEngine(m, n, k, 0, 0, p=p, caller_workbuf=True)
        assert e.ok
        w = torch.empty(e.workbuf_bytes + 256, dtype=torch.uint8, device="cuda")
        e.attach_workbuf((w.data_ptr() + 255) // 256 * 256)
        assert e.set_gemm_mode(cb.GEMM_PLAIN) == 0
        dC = dev_zeros(m * n)
        assert e.exec(dA, lda, dB, ldb, dC, m) == 0
        outs.append(from_dev(dC, m, n))
        e.free()
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])
