"""Asynchronous and captured execs whose operands change from call to call: queued
behind work that still runs, between synchronous calls, captured before the engine
ever ran, replayed between direct calls.  Every C has the bits of a synchronous
call on an engine of its own."""
import ctypes

import numpy as np
import pytest

import ca3dmm_b200 as cb
from oracle import oracle as orc
from tests._util import dev_zeros, from_dev, to_dev

pytestmark = pytest.mark.gpu

MODES = {"plain": cb.GEMM_PLAIN, "slices": cb.GEMM_OZAKI, "modular": cb.GEMM_CRT}
COUNT = {"plain": 0, "slices": 7, "modular": 15}
# tiles cut between CTAs; whole tiles, packed operands
SHAPES = [(300, 260, 700, 0, 0, 2), (257, 131, 333, 1, 1, 4)]


def _engine(m, n, k, ta, tb, p, mode):
    e = cb.Ca3dmmEngine(m, n, k, ta, tb, p=p)
    assert e.ok
    if mode != "plain":
        assert e.set_gemm_mode(MODES[mode], COUNT[mode]) == 0
    return e


def _sets(m, n, k, ta, tb, p, mode, count=3):
    """`count` operand pairs with their C buffers and the C each is to give."""
    out = []
    for i in range(count):
        dA, lda = to_dev(orc.gen_signed_exp(30 + i, *((k, m) if ta else (m, k))))
        dB, ldb = to_dev(orc.gen_signed_exp(60 + i, *((n, k) if tb else (k, n))))
        e, dC = _engine(m, n, k, ta, tb, p, mode), dev_zeros(m * n)
        assert e.exec(dA, lda, dB, ldb, dC, m) == 0
        out.append((dA, lda, dB, ldb, dC, m, from_dev(dC, m, n)))
        e.free()
        dC.zero_()
    return out


def _check(sets, m, n, which):
    import torch
    for i in which:
        assert np.array_equal(from_dev(sets[i][4], m, n), sets[i][6]), i
        sets[i][4].zero_()
    torch.cuda.synchronize()


@pytest.mark.parametrize("mode", sorted(MODES))
@pytest.mark.parametrize("m,n,k,ta,tb,p", SHAPES)
def test_queued_execs_with_changing_operands(cuda, mode, m, n, k, ta, tb, p):
    import torch
    sets = _sets(m, n, k, ta, tb, p, mode)
    e = _engine(m, n, k, ta, tb, p, mode)
    s = torch.cuda.Stream()
    for warm in (False, True):
        e.set_stream(s.cuda_stream, 0)
        with torch.cuda.stream(s):
            torch.cuda._sleep(20_000_000)            # about 10 ms
        for x in (sets[0], sets[1], sets[2], sets[0]):
            assert e.exec(*x[:6]) == 0
        if warm:                                     # a synchronous call behind them
            e.set_stream(s.cuda_stream, 1)
            assert e.exec(*sets[1][:6]) == 0
        torch.cuda.synchronize()
        _check(sets, m, n, (0, 1, 2))
    e.free()


@pytest.mark.parametrize("mode", sorted(MODES))
@pytest.mark.parametrize("m,n,k,ta,tb,p", SHAPES)
def test_captured_execs_between_direct_ones(cuda, mode, m, n, k, ta, tb, p):
    import torch
    sets = _sets(m, n, k, ta, tb, p, mode)
    e = _engine(m, n, k, ta, tb, p, mode)
    s = torch.cuda.Stream()
    graphs = []
    for i in (0, 1):                                 # captured before any direct call
        e.set_stream(s.cuda_stream, 0)
        g = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(g, stream=s):
            assert e.exec(*sets[i][:6]) == 0
        graphs.append(g)
        e.set_stream(s.cuda_stream, 1)               # the captured plan has not been uploaded
        assert e.exec(*sets[i][:6]) == 0
        _check(sets, m, n, (i,))
    for _ in range(2):
        assert e.exec(*sets[2][:6]) == 0
        with torch.cuda.stream(s):
            graphs[0].replay()
            graphs[1].replay()
        assert e.exec(*sets[2][:6]) == 0
        torch.cuda.synchronize()
        _check(sets, m, n, (0, 1, 2))
    graphs.clear()
    e.free()


@pytest.mark.parametrize("mode", sorted(MODES))
def test_grouped_execs_with_changing_operands(cuda, mode):
    import torch
    shapes = [(200, 150, 300), (64, 257, 129)]
    ms, ns, ks = zip(*shapes)
    mk = lambda: cb.GroupedGemm(ms, ns, ks, mode=MODES[mode], slices=COUNT[mode])
    sets, want = [], []
    for i in range(3):
        A = [to_dev(orc.gen_signed_exp(10 * i + j, m, k))[0] for j, (m, n, k) in enumerate(shapes)]
        B = [to_dev(orc.gen_signed_exp(10 * i + j + 5, k, n))[0] for j, (m, n, k) in enumerate(shapes)]
        Cs = [dev_zeros(m * n) for m, n, _ in shapes]
        x = (A, list(ms), B, list(ks), Cs, list(ms))
        g = mk()
        assert g.ok and g.exec(*x) == 0
        sets.append(x)
        want.append([c.cpu().numpy() for c in Cs])
        for c in Cs:
            c.zero_()

    def check(which):
        torch.cuda.synchronize()
        for i in which:
            for c, w in zip(sets[i][4], want[i]):
                assert np.array_equal(c.cpu().numpy(), w), i
                c.zero_()
        torch.cuda.synchronize()
    g, s = mk(), torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    g.set_stream(s.cuda_stream, 0)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=s):          # captured before any direct call
        assert g.exec(*sets[0]) == 0
    g.set_stream(s.cuda_stream, 1)
    assert g.exec(*sets[0]) == 0
    check((0,))
    g.set_stream(s.cuda_stream, 0)
    with torch.cuda.stream(s):
        torch.cuda._sleep(20_000_000)
    for x in sets:
        assert g.exec(*x) == 0
    check((0, 1, 2))
    for _ in range(2):
        assert g.exec(*sets[2]) == 0
        with torch.cuda.stream(s):
            graph.replay()
        assert g.exec(*sets[2]) == 0
        check((0, 2))
    del graph


def test_asynchronous_failure_is_not_the_next_calls(cuda, monkeypatch, capfd):
    """An asynchronous exec that finds a guard band overwritten reports it in its own
    status word, printed by the next synchronous exec, which succeeds."""
    import torch
    monkeypatch.setenv("CA3DMM_CANARY", "1")
    m, n, k = 300, 260, 700
    dA, lda = to_dev(orc.gen_signed_exp(3, m, k))
    dB, ldb = to_dev(orc.gen_signed_exp(4, k, n))
    dC = dev_zeros(m * n)
    e = cb.Ca3dmmEngine(m, n, k, 0, 0, p=2, caller_workbuf=True)
    w = torch.zeros(e.workbuf_bytes + 256, dtype=torch.uint8, device="cuda")
    base = (-w.data_ptr()) % 256
    e.attach_workbuf(w.data_ptr() + base)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    e.set_stream(s.cuda_stream, 1)
    assert e.exec(dA, lda, dB, ldb, dC, m) == 0
    off = (ctypes.c_longlong * 2)()
    assert cb.lib().ca3dmm_engine_guard_bands(e.e, off, 2) > 1
    band = w[base + off[1]:][:256]
    with torch.cuda.stream(s):
        torch.cuda._sleep(20_000_000)
        kept = band.clone()
        band.zero_()
        e.set_stream(s.cuda_stream, 0)
        assert e.exec(dA, lda, dB, ldb, dC, m) == 0
        band.copy_(kept)
    e.set_stream(s.cuda_stream, 1)
    capfd.readouterr()
    assert e.exec(dA, lda, dB, ldb, dC, m) == 0
    assert "Device status 6 of an earlier asynchronous exec" in capfd.readouterr().err
    assert e.exec(dA, lda, dB, ldb, dC, m) == 0
    assert "earlier" not in capfd.readouterr().err
    e.free()
