"""B^T B in the modular mode computes C's upper block triangle and mirrors it:
bit for bit the oracle's full product, for tile edges on both widths, several
slabs, bands of the work list, and host buffers."""
import numpy as np
import pytest

import ca3dmm_b200 as cb
from oracle import oracle as orc
from tests._util import dev_zeros, from_dev, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile_n", [256, 128])
@pytest.mark.parametrize("n,k,kp,band", [
    (1, 40, 1, 32), (128, 200, 1, 32), (129, 300, 2, 32), (200, 777, 3, 1), (257, 500, 1, 2),
    (385, 640, 2, 3), (512, 1000, 4, 32), (900, 333, 1, 2),
])
def test_upper_triangle(cuda, monkeypatch, tile_n, n, k, kp, band):
    import torch
    monkeypatch.setenv("CA3DMM_CRT_TILE_N", str(tile_n))
    monkeypatch.setenv("CA3DMM_CRT_BAND", str(band))
    B = orc.gen_btb(3, k, n)
    e = cb.Ca3dmmEngine(n, n, k, p=kp, btb=True, proc_grid=(1, 1, kp))
    assert e.ok and e.set_gemm_mode(cb.GEMM_CRT, 15) == 0
    dB, ldb = to_dev(B)
    dC = dev_zeros(n * n).fill_(-1.0)
    assert e.exec(None, 0, dB, ldb, dC, n) == 0
    got = from_dev(dC, n, n)
    want = None
    Bt = np.asfortranarray(B.T)
    for s in range(kp):
        k0, kz = orc.block_spos_size(k, kp, s)
        c = orc.crt_gemm(np.asfortranarray(Bt[:, k0:k0 + kz]), np.asfortranarray(B[k0:k0 + kz, :]),
                         0, 0, n, n, kz, orc.crt_bits(15, kz))
        want = c if want is None else want + c
    assert np.array_equal(got, want)
    hB = torch.from_numpy(np.asfortranarray(B).ravel(order="F").copy()).pin_memory()
    hC = torch.zeros(n * n, dtype=torch.float64).pin_memory()
    assert e.exec_host(None, 0, hB, ldb, hC, n) == 0
    assert np.array_equal(hC.numpy().reshape(n, n).T, want)
    e.free()
