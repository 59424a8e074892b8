"""The numbering of the run copies' work items, checked on the CPU; runs that are
almost as long as a 32-bit count, copied on the GPU."""
import ctypes as C
import random

import pytest

import ca3dmm_b200 as cb

INT_MAX = 2 ** 31 - 1


class Piece(C.Structure):
    _fields_ = [("src", C.c_void_p), ("dst", C.c_void_p)] + [
        (n, C.c_int) for n in ("lds", "ldd", "len", "runs")]


def pieces(shapes):
    """shapes: [(len, runs)]"""
    P = (Piece * max(1, len(shapes)))()
    for p, (length, runs) in zip(P, shapes):
        p.lds = p.ldd = p.len = length
        p.runs = runs
    return P


def items(shapes):
    L = cb.lib()
    L.ca3dmm_copy_runs_items.restype = C.c_longlong
    return L.ca3dmm_copy_runs_items(pieces(shapes), len(shapes))


@pytest.mark.parametrize("length", [INT_MAX - 4096, INT_MAX - 2048, INT_MAX - 600, INT_MAX - 500,
                                    INT_MAX - 60, INT_MAX])
@pytest.mark.parametrize("turn", [False, True])
def test_counts_near_the_limit(length, turn):
    """A launch has items for all of a run, or is refused: never none."""
    got = items([(1, length) if turn else (length, 1)])
    assert got == -1 or got * (2048 if turn else 512) >= length


def test_no_items_of_empty_pieces():
    assert items([]) == 0 and items([(0, 5), (5, 0)]) == 0


def layouts():
    rng = random.Random(5)
    out = [[(1, 1)], [(333, 7)] * 24, [(20, 1600), (33, 3), (512, 1), (1, 1)],
           [(8000, 8000)] + [(20, 10)] * 400, [(8, 3900)] + [(8, 1)] * 511,
           [(334, 7981)] * 24 + [(334, 1)] * 456, [(40000, 3), (0, 4), (4, 0), (17, 90)]]
    for _ in range(30):
        n = rng.choice([1, 2, 63, 64, 65, 200, 512])
        top = rng.choice([4, 40, 400, 4000])
        out.append([(rng.randint(0, top), rng.randint(0, max(1, 3000 // top))) for _ in range(n)])
    return out


@pytest.mark.parametrize("shapes", layouts(), ids=lambda s: "%dx" % len(s))
def test_items_cover_every_run_once(shapes):
    """Every column of every run, wherever in a line it starts, in one item; at most a
    fifth of the items are empty turns."""
    L = cb.lib()
    P, n, out = pieces(shapes), items(shapes), (C.c_int * 5)()
    full = [s for s in shapes if s[0] > 0 and s[1] > 0]
    seen = [{} for _ in full]
    empty = 0
    for i in range(n):
        assert L.ca3dmm_copy_runs_item(P, len(shapes), C.c_longlong(i), out) == 0
        k, r0, r1, c0, c1 = out
        if r0 == r1:
            empty += 1
            continue
        assert 0 <= r0 < r1 <= full[k][1] and 0 <= c0 < c1
        seen[k].setdefault((r0, r1), []).append((c0, c1))
    for (length, runs), got in zip(full, seen):
        spans = sorted(got)
        assert [a for a, _ in spans] == [0] + [b for _, b in spans[:-1]] and spans[-1][1] == runs
        for chunks in got.values():
            chunks.sort()
            assert chunks[0][0] == 0 and all(a[1] == b[0] for a, b in zip(chunks, chunks[1:]))
            assert chunks[-1][1] == length + 15
    assert empty <= 0.2 * n
    assert L.ca3dmm_copy_runs_item(P, len(shapes), C.c_longlong(n), out) != 0


def rects(heights, widths, r0=0):
    out = []
    for h in heights:
        c0 = 0
        for w in widths:
            out.append((r0, c0, h, w))
            c0 += w
        r0 += h
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("src,dst", [
    (rects([3001], [77, 400, 5, 900]), rects([2990] + [1] * 11, [1382])),
    (rects([60], [8000]), rects([10], [20] * 400) + rects([50], [8000], 10)),
    (rects([5000], [8]), rects([1] * 20 + [4900] + [1] * 80, [8])),
    (rects([700], [33, 64, 20, 31, 127, 129, 240, 3]), rects([1, 699], [300, 347])),
])
def test_uneven_layouts(cuda, src, dst):
    import torch
    rows, cols = max(r + h for r, _, h, _ in src), max(c + w for _, c, _, w in src)
    G = torch.rand(rows, cols, dtype=torch.float64, device="cuda")
    cut = lambda R: [G[r:r + h, c:c + w].contiguous() for r, c, h, w in R]
    S, want = cut(src), cut(dst)
    D = [torch.full_like(w, -7.0) for w in want]
    lay = cb.RedistLayouts(src, dst)
    assert lay.ok and lay.exec(S, [x.shape[1] for x in S], D, [x.shape[1] for x in D]) == 0
    assert all(torch.equal(a, b) for a, b in zip(D, want))


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


@pytest.mark.gpu
@pytest.mark.parametrize("strips,pr,pc", [(64, 9, 10), (7, 3, 2)])    # more than 512 pieces, fewer
def test_two_streams(cuda, strips, pr, pc):
    """One handle on two streams, the first held up: each exec moves its own blocks."""
    import torch
    n = 640
    cut = lambda p: [(n * i // p, n * (i + 1) // p - n * i // p) for i in range(p)]
    src = [(0, c0, n, w) for c0, w in cut(strips)]
    dst = [(r0, c0, h, w) for r0, h in cut(pr) for c0, w in cut(pc)]
    lay = cb.RedistLayouts(src, dst)
    assert lay.ok
    sets = []
    for _ in range(2):
        G = torch.rand(n, n, dtype=torch.float64, device="cuda")
        blocks = lambda R: [G[r:r + h, c:c + w].contiguous() for r, c, h, w in R]
        S, want = blocks(src), blocks(dst)
        sets.append((S, [torch.zeros_like(w) for w in want], want, torch.cuda.Stream()))
    torch.cuda.synchronize()
    with torch.cuda.stream(sets[0][3]):
        torch.cuda._sleep(20_000_000)
    for S, D, _, s in sets:
        assert lay.exec(S, [x.shape[1] for x in S], D, [x.shape[1] for x in D], s.cuda_stream) == 0
    torch.cuda.synchronize()
    for _, D, want, _ in sets:
        assert all(torch.equal(a, b) for a, b in zip(D, want))
