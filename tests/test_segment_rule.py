"""Which products the k segments cut: those that equal shares shorten by more than the
cutting costs.  Read off the plan on the CPU."""
import ctypes as C

import pytest

import ca3dmm_b200 as cb


class Seg(C.Structure):
    _fields_ = [(n, C.c_int) for n in ("tm", "tn", "kt0", "kt1", "part", "nparts", "slot0", "counter")]


def cut_tiles(m, n, k):
    """Tiles in more than one part; None when whole tiles go to the grouped kernel."""
    L = cb.lib()
    mx = L.ca3dmm_dgemm_segments_max(m, n, k)
    if mx == 0:
        return None
    segs, order, begin = (Seg * mx)(), (C.c_int * mx)(), (C.c_int * 149)()
    ns, grid, nc = C.c_int(), C.c_int(), C.c_int()
    assert L.ca3dmm_dgemm_segments(m, n, k, 128, segs, order, begin, C.byref(ns), C.byref(grid),
                                   C.byref(nc)) == 0
    return nc.value


# measured both ways: cutting these is slower
@pytest.mark.parametrize("m,n,k", [
    (1408, 1408, 256), (1664, 1280, 256), (1408, 1408, 512), (1152, 1280, 96), (1536, 1408, 512),
    (4736, 1024, 2048), (128, 128, 64),
])
def test_left_whole(m, n, k):
    assert cut_tiles(m, n, k) == 0


@pytest.mark.parametrize("m,n,k", [
    (200, 150, 300), (1000, 1000, 1000), (768, 768, 768), (2048, 2048, 2048), (3200, 3200, 3200),
    (2432, 4096, 1000), (3200, 3100, 500), (1501, 2003, 3001),
])
def test_cut(m, n, k):
    assert cut_tiles(m, n, k) > 0


@pytest.mark.parametrize("m,n,k", [(5000, 5000, 5000), (8000, 8000, 8000), (4736, 3072, 4000)])
def test_many_rounds_stay_with_the_grouped_kernel(m, n, k):
    assert cut_tiles(m, n, k) is None


@pytest.mark.parametrize("m,n,k", [
    (200, 150, 300), (1000, 1000, 1000), (768, 768, 768), (2048, 2048, 2048), (1408, 1408, 256),
    (129, 131, 257), (640, 700, 4097), (1501, 2003, 3001), (3200, 3100, 500), (128, 128, 100000),
    (2500, 1300, 777), (5000, 640, 33), (300, 260, 700), (1, 1, 9999),
])
def test_partials_hold_the_cut_tiles_and_no_more(m, n, k):
    L = cb.lib()
    L.ca3dmm_dgemm_segments_ws_bytes.restype = C.c_size_t
    mx = L.ca3dmm_dgemm_segments_max(m, n, k)
    segs, order, begin = (Seg * mx)(), (C.c_int * mx)(), (C.c_int * 149)()
    ns, grid, nc = C.c_int(), C.c_int(), C.c_int()
    for tile_n in (128, 64):
        assert L.ca3dmm_dgemm_segments(m, n, k, tile_n, segs, order, begin, C.byref(ns),
                                       C.byref(grid), C.byref(nc)) == 0
        need = sum(1 for s in segs[:ns.value] if s.nparts > 1) * 128 * tile_n * 8
        got = L.ca3dmm_dgemm_segments_ws_bytes(m, n, k)
        assert got == need if tile_n == 128 else got >= need
