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
