"""The numbering of the run copies' work items, checked on the CPU; runs that are
almost as long as a 32-bit count, copied on the GPU."""
import ctypes as C

import pytest

import ca3dmm_b200 as cb

INT_MAX = 2 ** 31 - 1


class Piece(C.Structure):
    _fields_ = [("src", C.c_void_p), ("dst", C.c_void_p)] + [
        (n, C.c_int) for n in ("lds", "ldd", "len", "runs")]


def items(shapes):
    """shapes: [(len, runs)]"""
    L = cb.lib()
    L.ca3dmm_copy_runs_items.restype = C.c_longlong
    P = (Piece * max(1, len(shapes)))()
    for p, (length, runs) in zip(P, shapes):
        p.lds = p.ldd = p.len = length
        p.runs = runs
    return L.ca3dmm_copy_runs_items(P, len(shapes))


@pytest.mark.parametrize("length", [INT_MAX - 4096, INT_MAX - 2048, INT_MAX - 600, INT_MAX - 500,
                                    INT_MAX - 60, INT_MAX])
@pytest.mark.parametrize("turn", [False, True])
def test_counts_near_the_limit(length, turn):
    """A launch has items for all of a run, or is refused: never none."""
    got = items([(1, length) if turn else (length, 1)])
    assert got == -1 or got * (4 if turn else 512) >= length


def test_no_items_of_empty_pieces():
    assert items([]) == 0 and items([(0, 5), (5, 0)]) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("length", [INT_MAX - 3000, INT_MAX - 300, INT_MAX])
def test_longest_runs(cuda, length):
    import torch
    if torch.cuda.mem_get_info()[0] < 2 * 8 * length + (4 << 30):
        pytest.skip("needs 36 GB of free device memory")
    src = torch.arange(length, dtype=torch.float64, device="cuda")
    dst = torch.zeros(length, dtype=torch.float64, device="cuda")
    lay = cb.RedistLayouts([(0, 0, 1, length)], [(0, 0, 1, length)])
    assert lay.ok and lay.exec([src], [length], [dst], [length]) == 0
    same = all(torch.equal(a, b) for a, b in zip(src.split(1 << 28), dst.split(1 << 28)))
    del src, dst
    torch.cuda.empty_cache()
    assert same
