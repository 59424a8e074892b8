"""The work that users of this library have it do, as cases that can be timed.

Each case goes through the public entry points of ``ca3dmm_b200``: an engine
exec in one of its GEMM modes, the tall-skinny Gram product, a batch of uneven
GEMMs in one grouped call, a redistribution between two layouts.  ``prepare``
makes what a program holds before the call (device operands, the engine or
batch handle, the output buffer); ``run`` is the one call that the program
repeats.

Matrices are column-major.  A column-major r x c matrix with leading dimension
r is held as the row-major torch tensor of shape (c, r).
"""
import math

import torch

import ca3dmm_b200 as cb

MODES = {"plain": cb.GEMM_PLAIN, "slices": cb.GEMM_OZAKI, "modular": cb.GEMM_CRT}


def engine(name, m, n, k, ta, tb, p, mode, count, entries, grid=""):
    """C = op(A) op(B) through ca3dmm_engine_exec on p virtual ranks.

    count: INT8 slices, or moduli (0: the library's choice); entries:
    "uniform" in [-1, 1) or "spread" (sign (1 + u) 2^e, e in [-8, 8]).
    """
    c = {"kind": "engine", "m": m, "n": n, "k": k, "ta": ta, "tb": tb, "p": p, "grid": grid,
         "mode": mode, "count": count, "entries": entries}
    return dict(c, name=name) if name else c


def gram(name, n, k, p, mode):
    c = {"kind": "gram", "n": n, "k": k, "p": p, "mode": mode}
    return dict(c, name=name) if name else c


def grouped(name, batch, lo, hi, mode, shapes):
    c = {"kind": "grouped", "batch": batch, "lo": lo, "hi": hi, "mode": mode, "shapes": shapes}
    return dict(c, name=name) if name else c


def redist(name, rows, cols, strips, pr, pc):
    c = {"kind": "redist", "rows": rows, "cols": cols, "strips": strips, "pr": pr, "pc": pc}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest products a caller's loop makes: launches and host time count
        engine("plain_small", 200, 150, 300, 0, 0, 4, "plain", 0, "uniform"),
        # one block of a blocked solver: fewer output tiles than the chip has SMs
        engine("plain_1000", 1000, 1000, 1000, 0, 0, 1, "plain", 0, "spread"),
        # the example driver's size: uniform entries, four ranks
        engine("plain_2048", 2048, 2048, 2048, 0, 0, 4, "plain", 0, "uniform"),
        # odd sizes with both operands transposed: nothing is aligned for TMA
        engine("plain_ragged_tt", 1501, 2003, 3001, 1, 1, 6, "plain", 0, "spread"),
        # the benchmark's square product on its 24-rank grid, native FP64
        engine("plain_8000", 8000, 8000, 8000, 0, 0, 24, "plain", 0, "spread", "4x2x3"),
        # split precision where its passes over the operands and C weigh as much as the GEMM
        engine("modular_2048", 2048, 2048, 2048, 0, 0, 4, "modular", 0, "uniform"),
        # the same with odd sizes, both operands transposed and a deeper k
        engine("modular_ragged_tt", 1999, 1201, 4099, 1, 1, 6, "modular", 0, "spread"),
        # the benchmark's square product in its headline mode
        engine("modular_8000", 8000, 8000, 8000, 0, 0, 24, "modular", 0, "spread", "4x2x3"),
        # the other split precision mode (seven INT8 slices), a middle size
        engine("slices_4000", 4000, 4000, 4000, 0, 0, 8, "slices", 7, "spread"),
        # the Gram step of CholeskyQR: tall and skinny, columns scaled over six decades
        gram("gram_modular", 512, 1048576, 32, "modular"),
        # a batch of uneven independent products in one grouped call
        grouped("grouped_modular", 256, 64, 4096, "modular", 2024),
        # 1D column strips to a 2D block layout, every rank's blocks in one call
        redist("redist_8000", 8000, 8000, 24, 4, 6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _engine_draw(rng, mode, top):
    # sizes as the autotuner's study draws them, up to the largest listed product
    while True:
        m, n, k = (_log_int(rng, 128, 16384) for _ in range(3))
        if m * n * k <= top ** 3 and 8 * (m * n + m * k + n * k) <= 24 * 8000 ** 2:
            break
    count = {"plain": 0, "modular": rng.choice([0, 0, 0, 14, 16]),
             "slices": rng.choice([6, 7, 7, 8])}[mode]
    return engine("", m, n, k, rng.randint(0, 1), rng.randint(0, 1), rng.choice([1, 4, 6, 8, 24]),
                  mode, count, rng.choice(["uniform", "spread"]))


def draw(rng):
    kind = rng.choice(["plain", "plain", "plain", "modular", "modular", "modular", "slices", "gram",
                       "grouped", "redist"])
    if kind == "plain" or kind == "modular":
        return _engine_draw(rng, kind, 8000)
    if kind == "slices":
        return _engine_draw(rng, kind, 4000)
    if kind == "gram":
        return gram("", _log_int(rng, 64, 512), _log_int(rng, 65536, 1048576),
                    rng.choice([16, 24, 32]), rng.choice(["plain", "modular"]))
    if kind == "grouped":
        return grouped("", rng.randint(8, 224), 64, rng.choice([512, 1024, 2048]),
                       rng.choice(["plain", "modular"]), rng.randrange(1 << 20))
    return redist("", _log_int(rng, 500, 8000), _log_int(rng, 500, 8000), rng.randint(1, 24),
                  rng.randint(1, 4), rng.randint(1, 6))


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _matrix(g, r, c, entries):
    """A column-major r x c matrix, as the (c, r) tensor."""
    u = torch.rand(c, r, dtype=torch.float64, device="cuda", generator=g)
    if entries == "uniform":
        return u.mul_(2.0).sub_(1.0)
    lo, hi = (-8, 8) if entries == "spread" else (-4, 4)
    e = torch.randint(lo, hi + 1, (c, r), dtype=torch.int32, device="cuda", generator=g)
    if entries == "spread":
        s = torch.randint(0, 2, (c, r), dtype=torch.int8, device="cuda", generator=g)
        return torch.ldexp(u.add_(1.0), e).mul_(s.mul_(2).sub_(1))
    return torch.ldexp(u.mul_(2.0).sub_(1.0), e)


def _engine_operands(c, seed):
    g = _gen(seed)
    m, n, k = c["m"], c["n"], c["k"]
    A = _matrix(g, *((k, m) if c["ta"] else (m, k)), c["entries"])
    B = _matrix(g, *((n, k) if c["tb"] else (k, n)), c["entries"])
    return A, B


def _gram_operand(c, seed):
    g = _gen(seed)
    z = torch.randn(c["n"], c["k"], dtype=torch.float64, device="cuda", generator=g)
    u = torch.rand(c["n"], dtype=torch.float64, device="cuda", generator=g) * 6.0 - 3.0
    return z.mul_(torch.pow(10.0, u)[:, None])


def _grouped_sizes(c):
    import random
    rng = random.Random(c["shapes"])
    return [tuple(_log_int(rng, c["lo"], c["hi"]) for _ in range(3)) +
            (rng.randint(0, 1), rng.randint(0, 1)) for _ in range(c["batch"])]


def _grouped_operands(c, seed):
    g = _gen(seed)
    As, Bs = [], []
    for m, n, k, ta, tb in _grouped_sizes(c):
        As.append(_matrix(g, *((k, m) if ta else (m, k)), "batch"))
        Bs.append(_matrix(g, *((n, k) if tb else (k, n)), "batch"))
    return As, Bs


def _splits(length, parts):
    return [cb.calc_block_spos_size(length, parts, i) for i in range(parts)]


def _even_splits(length, parts):
    """calc_block_spos_size's balanced split, restated (the longer blocks first)."""
    q, r = divmod(length, parts)
    return [((q + 1) * i, q + 1) if i < r else (q * i + r, q) for i in range(parts)]


def _redist_source(c, seed):
    return torch.rand(c["rows"], c["cols"], dtype=torch.float64, device="cuda", generator=_gen(seed))


# ---------------------------------------------------------------- the cases
def prepare(case, seed):
    kind = case["kind"]
    if kind == "engine":
        A, B = _engine_operands(case, seed)
        m, n, k = case["m"], case["n"], case["k"]
        grid = tuple(int(x) for x in case["grid"].split("x")) if case["grid"] else None
        eng = cb.Ca3dmmEngine(m, n, k, case["ta"], case["tb"], p=case["p"], proc_grid=grid)
        if not eng.ok or (case["mode"] != "plain" and
                          eng.set_gemm_mode(MODES[case["mode"]], case["count"])):
            raise RuntimeError("engine set-up failed")
        C = torch.zeros(n, m, dtype=torch.float64, device="cuda")
        return {"kind": kind, "eng": eng, "A": A, "B": B, "C": C, "lda": A.shape[1],
                "ldb": B.shape[1], "ldc": m}
    if kind == "gram":
        B = _gram_operand(case, seed)
        eng = cb.Ca3dmmEngine(case["n"], case["n"], case["k"], p=case["p"],
                              proc_grid=(1, 1, case["p"]), btb=True)
        if not eng.ok or (case["mode"] != "plain" and eng.set_gemm_mode(MODES[case["mode"]], 0)):
            raise RuntimeError("engine set-up failed")
        C = torch.zeros(case["n"], case["n"], dtype=torch.float64, device="cuda")
        return {"kind": kind, "eng": eng, "B": B, "C": C, "ldb": case["k"], "ldc": case["n"]}
    if kind == "grouped":
        As, Bs = _grouped_operands(case, seed)
        ms, ns, ks, tas, tbs = zip(*_grouped_sizes(case))
        handle = cb.GroupedGemm(ms, ns, ks, tas, tbs, mode=MODES[case["mode"]], slices=0)
        if not handle.ok:
            raise RuntimeError("batch set-up failed")
        # every C starts on a 16-byte boundary of one buffer, as a caller's arena places them
        sizes = [(m * n + 1) // 2 * 2 for m, n in zip(ms, ns)]
        C = torch.zeros(sum(sizes), dtype=torch.float64, device="cuda")
        Cs = list(torch.split(C, sizes))
        return {"kind": kind, "batch": handle, "A": As, "B": Bs, "C": C, "Cs": Cs,
                "lda": [a.shape[1] for a in As], "ldb": [b.shape[1] for b in Bs], "ldc": list(ms)}
    X = _redist_source(case, seed)
    src, dst, s_rects, d_rects = [], [], [], []
    for c0, w in _splits(case["cols"], case["strips"]):
        s_rects.append((0, c0, case["rows"], w))
        src.append(X[:, c0:c0 + w].contiguous())
    for r0, h in _splits(case["rows"], case["pr"]):
        for c0, w in _splits(case["cols"], case["pc"]):
            d_rects.append((r0, c0, h, w))
            dst.append(torch.zeros(h, w, dtype=torch.float64, device="cuda"))
    lay = cb.RedistLayouts(s_rects, d_rects)
    if not lay.ok:
        raise RuntimeError("layout set-up failed")
    return {"kind": kind, "lay": lay, "src": src, "dst": dst,
            "src_ld": [x.shape[1] for x in src], "dst_ld": [x.shape[1] for x in dst]}


def run(state):
    kind = state["kind"]
    if kind == "engine":
        rc = state["eng"].exec(state["A"], state["lda"], state["B"], state["ldb"], state["C"],
                               state["ldc"])
        out = state["C"]
    elif kind == "gram":
        rc = state["eng"].exec(None, 0, state["B"], state["ldb"], state["C"], state["ldc"])
        out = state["C"]
    elif kind == "grouped":
        rc = state["batch"].exec(state["A"], state["lda"], state["B"], state["ldb"], state["Cs"],
                                 state["ldc"])
        out = state["C"]
    else:
        rc = state["lay"].exec(state["src"], state["src_ld"], state["dst"], state["dst_ld"])
        out = state["dst"]
    if rc:
        raise RuntimeError("call failed: %d" % rc)
    return out


def work(case):
    kind = case["kind"]
    if kind == "engine":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 8 * (m * k + k * n + m * n), "flops": 2 * m * n * k}
    if kind == "gram":
        n, k = case["n"], case["k"]
        return {"bytes": 8 * (n * k + n * n), "flops": 2 * n * n * k}
    if kind == "grouped":
        s = _grouped_sizes(case)
        return {"bytes": sum(8 * (m * k + k * n + m * n) for m, n, k, _, _ in s),
                "flops": sum(2 * m * n * k for m, n, k, _, _ in s)}
    return {"bytes": 16 * case["rows"] * case["cols"], "flops": 0}


# ---------------------------------------------------------------- reference values
def _product(X, Y):
    """X @ Y in 64 bits: partial products over short ranges of k, added with the
    rounding errors of the additions carried along (Knuth's two-sum)."""
    k = X.shape[1]
    step = max(256, -(-k // 256))
    s = torch.zeros(X.shape[0], Y.shape[1], dtype=torch.float64, device="cuda")
    err = torch.zeros_like(s)
    for k0 in range(0, k, step):
        p = X[:, k0:k0 + step] @ Y[k0:k0 + step]
        t = s + p
        z = t - s
        err += (s - (t - z)) + (p - z)
        s = t
    return s + err


def exact(case, seed):
    kind = case["kind"]
    if kind == "engine":
        A, B = _engine_operands(case, seed)
        # C^T = op(B)^T op(A)^T; the (c, r) tensor of X is X^T
        return _product(B.t() if case["tb"] else B, A.t() if case["ta"] else A)
    if kind == "gram":
        B = _gram_operand(case, seed)
        return _product(B, B.t())
    if kind == "grouped":
        out = []
        As, Bs = _grouped_operands(case, seed)
        for (m, n, k, ta, tb), A, B in zip(_grouped_sizes(case), As, Bs):
            C = _product(B.t() if tb else B, A.t() if ta else A).reshape(-1)
            out.append(torch.cat([C, C.new_zeros((m * n) % 2)]))
        return torch.cat(out)
    X = _redist_source(case, seed)
    return [X[r0:r0 + h, c0:c0 + w].contiguous()
            for r0, h in _even_splits(case["rows"], case["pr"])
            for c0, w in _even_splits(case["cols"], case["pc"])]
