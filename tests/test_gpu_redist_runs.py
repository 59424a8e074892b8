"""mat_redist_layouts_exec where the pieces travel with the launch (up to 512 of
them) and where they do not: runs of one element to several chunks, odd widths
and leading dimensions, an asynchronous stream; bit for bit against slicing."""
import numpy as np
import pytest

import ca3dmm_b200 as cb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,strips,pr,pc,pad", [
    (1, 1, 1, 1, 1, 0), (3, 512, 1, 1, 1, 1), (6, 513, 1, 2, 1, 0), (5, 1025, 2, 1, 3, 3),
    (700, 333, 24, 4, 6, 0), (33, 4000, 3, 5, 2, 1),
    (100, 640, 64, 9, 10, 0),            # more than 512 pieces
])
@pytest.mark.parametrize("use_stream", [False, True])
def test_runs(cuda, rows, cols, strips, pr, pc, pad, use_stream):
    import torch
    G = torch.rand(rows, cols, dtype=torch.float64, device="cuda")
    cut = lambda n, p: [(n * i // p, n * (i + 1) // p - n * i // p) for i in range(p)]
    src_r = [(0, c0, rows, w) for c0, w in cut(cols, strips)]
    dst_r = [(r0, c0, h, w) for r0, h in cut(rows, pr) for c0, w in cut(cols, pc)]

    def block(r):
        b = torch.full((r[2], r[3] + pad), -7.0, dtype=torch.float64, device="cuda")
        return b
    src, dst = [], []
    for r in src_r:
        b = block(r)
        b[:, :r[3]] = G[r[0]:r[0] + r[2], r[1]:r[1] + r[3]]
        src.append(b)
    dst = [block(r) for r in dst_r]
    L = cb.RedistLayouts(src_r, dst_r)
    assert L.ok
    s = torch.cuda.Stream() if use_stream else None
    torch.cuda.synchronize()
    assert L.exec(src, [b.shape[1] for b in src], dst, [b.shape[1] for b in dst],
                  s.cuda_stream if s else None) == 0
    torch.cuda.synchronize()
    for r, b in zip(dst_r, dst):
        want = G[r[0]:r[0] + r[2], r[1]:r[1] + r[3]].cpu().numpy()
        got = b.cpu().numpy()
        assert np.array_equal(got[:, :r[3]], want)
        assert np.all(got[:, r[3]:] == -7.0)
