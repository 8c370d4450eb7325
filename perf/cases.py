"""Performance cases of the double-double BLAS: calls of its public entry points as a program makes them.

Every case is a plain dict. `prepare` makes its operands from a seed, `run` makes one call through the
ctypes binding (mwblas.py, the Fortran-style symbols), synchronous as the drop-in library is by default,
and returns the whole output array as its two limbs. `exact` is the same result from plain 64-bit torch;
it is good for the high limb only, so the low limb has no value there.

Values are those of the library's benchmark: hi ~ U[-1, 1), lo = hi * 2^-53 * U[-1, 1), renormalised;
where `fp64` is set, lo = 0 (a program that promotes double arrays). beta stays below one in magnitude,
so that a call repeated in place converges instead of overflowing.
"""
import importlib.util
import math
import os
import random

import numpy as np
import torch

_PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "epblas-parallel_gb300")
_LIBRARY = None


def _library():
    global _LIBRARY
    if _LIBRARY is None:
        spec = importlib.util.spec_from_file_location("mwblas", os.path.join(_PACKAGE, "mwblas.py"))
        module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(module)
        _LIBRARY = module.MWBlas(os.path.join(_PACKAGE, "libmwblas_gb300.so"))
    return _LIBRARY


# ---- the cases -------------------------------------------------------------------------------


def listed():
    return [
        # one small product on device arrays, as a blocked factorisation makes them in its panels:
        # launches and latency count
        dict(name="gemm_small", op="gemm", ta="N", tb="N", m=48, n=33, k=40, pad=0, beta=True, fp64=False),
        # the 512-cubed product handed over in ordinary host arrays, as a Fortran or C caller of the
        # drop-in symbol does; alpha = 1, beta = 0
        dict(name="gemm_host_512", op="gemm_host", ta="N", tb="N", m=512, n=512, k=512, beta=False),
        # an ordinary product with odd sizes, one operand transposed, padded leading dimensions
        dict(name="gemm_ragged", op="gemm", ta="T", tb="N", m=1531, n=1277, k=2011, pad=5, beta=True, fp64=False),
        # the headline product
        dict(name="gemm_8192", op="gemm", ta="N", tb="N", m=8192, n=8192, k=8192, pad=0, beta=True, fp64=False),
        # complex product with a conjugate transpose, odd sizes
        dict(name="wgemm", op="wgemm", ta="N", tb="C", m=2049, n=1900, k=2300),
        # symmetric rank-k update (the trailing update of a Cholesky factorisation)
        dict(name="syrk", op="syrk", uplo="U", trans="N", n=8192, k=2048),
        # triangular solve with many right-hand sides (the panel solve of a factorisation)
        dict(name="trsm", op="trsm", side="L", uplo="L", trans="N", diag="N", m=4096, n=1024),
        # matrix-vector product over a matrix far beyond the caches (one step of an iterative solver)
        dict(name="gemv_n", op="gemv", trans="N", m=16384, n=16384, pad=0),
        # the transposed product with odd sizes and a padded leading dimension
        dict(name="gemv_t", op="gemv", trans="T", m=7001, n=5003, pad=3),
        # inner product of long vectors: the result comes back to the host
        dict(name="dot", op="dot", n=100000000),
        # vector update, medium length
        dict(name="axpy", op="axpy", n=10000019),
        # a batch of uneven small products in one call
        dict(name="grouped", op="grouped", count=4000, low=8, high=512, shape_seed=1),
    ]


def _log(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    op = rng.choice(["gemm", "gemm", "gemm", "gemm_host", "wgemm", "syrk", "trsm", "trsm", "gemv", "gemv", "dot",
                     "axpy", "grouped"])
    if op == "gemm":
        return dict(op=op, ta=rng.choice("NT"), tb=rng.choice("NT"), m=_log(rng, 16, 8191), n=_log(rng, 16, 8191),
                    k=_log(rng, 16, 8191), pad=rng.choice([0, 1, 8]), beta=rng.random() < 0.7,
                    fp64=rng.random() < 0.2)
    if op == "gemm_host":
        return dict(op=op, ta=rng.choice("NT"), tb=rng.choice("NT"), m=_log(rng, 32, 1024), n=_log(rng, 32, 1024),
                    k=_log(rng, 32, 1024), beta=rng.random() < 0.5)
    if op == "wgemm":
        return dict(op=op, ta=rng.choice("NTC"), tb=rng.choice("NTC"), m=_log(rng, 64, 2500), n=_log(rng, 64, 2500),
                    k=_log(rng, 64, 2500))
    if op == "syrk":
        return dict(op=op, uplo=rng.choice("UL"), trans=rng.choice("NT"), n=_log(rng, 64, 8192),
                    k=_log(rng, 32, 2048))
    if op == "trsm":
        return dict(op=op, side=rng.choice("LR"), uplo=rng.choice("UL"), trans=rng.choice("NT"),
                    diag=rng.choice("NNU"), m=_log(rng, 64, 4096), n=_log(rng, 64, 4096))
    if op == "gemv":
        return dict(op=op, trans=rng.choice("NT"), m=_log(rng, 256, 16384), n=_log(rng, 256, 16384),
                    pad=rng.choice([0, 1, 3]))
    if op == "grouped":
        return dict(op=op, count=_log(rng, 300, 4000), low=8, high=rng.choice([128, 256, 512]),
                    shape_seed=rng.randrange(1 << 20))
    return dict(op=op, n=_log(rng, 1000, 100000000))


def _shapes(case):
    """The sizes (m, n, k) of a batch's instances: log-uniform in [low, high]."""
    rng = random.Random(case["shape_seed"])
    return [tuple(_log(rng, case["low"], case["high"]) for _ in range(3)) for _ in range(case["count"])]


# ---- inputs ----------------------------------------------------------------------------------


def _values(gen, shape, fp64=False):
    hi = torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64).mul_(2).sub_(1)
    out = torch.zeros((*shape, 2), device="cuda", dtype=torch.float64)
    if fp64:
        out[..., 0] = hi
        return out
    lo = torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64).mul_(2).sub_(1).mul_(hi).mul_(2.0 ** -53)
    out[..., 0] = hi + lo
    out[..., 1] = lo - (out[..., 0] - hi)
    return out


def _scalar(rng, low, high):
    v = rng.uniform(low, high) * rng.choice([-1.0, 1.0])
    return np.array([v, v * 2.0 ** -53 * rng.uniform(-0.9, 0.9)])


def _inputs(case, seed):
    """The operands of one call, column-major: element (i, j) of a matrix at [j, i]."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    rng = random.Random(seed)
    op, s = case["op"], {}
    s["alpha"], s["beta"] = _scalar(rng, 0.5, 2.0), _scalar(rng, 0.5, 0.95)
    if op in ("gemm", "gemm_host", "wgemm"):
        m, n, k, pad = case["m"], case["n"], case["k"], case.get("pad", 0)
        limbs = (2,) if op == "wgemm" else ()
        mats = []
        for rows, cols in ((m, k) if case["ta"] == "N" else (k, m), (k, n) if case["tb"] == "N" else (n, k), (m, n)):
            mats.append(_values(gen, (cols, rows + pad, *limbs), case.get("fp64", False)))
        s["a"], s["b"], s["c"] = mats
        if op == "wgemm":
            s["alpha"], s["beta"] = (np.stack([0.7 * v, 0.6 * v]) for v in (s["alpha"], s["beta"]))
        elif not case["beta"]:
            s["alpha"], s["beta"] = np.array([1.0, 0.0]), np.zeros(2)
    elif op == "syrk":
        n, k = case["n"], case["k"]
        s["a"] = _values(gen, (k, n) if case["trans"] == "N" else (n, k))
        s["c"] = _values(gen, (n, n))
    elif op == "trsm":
        order = case["m"] if case["side"] == "L" else case["n"]
        s["a"] = _values(gen, (order, order))
        if case["diag"] == "U":
            s["a"] /= 2.0 ** math.ceil(math.log2(order))
        else:   # diagonally dominant: diagonal uniform in [order, 2 order]
            diagonal = torch.rand(order, generator=gen, device="cuda", dtype=torch.float64).add_(1).mul_(order)
            s["a"][..., 0].diagonal().copy_(diagonal)
            s["a"][..., 1].diagonal().zero_()
        s["b"] = _values(gen, (case["n"], case["m"]))
    elif op == "gemv":
        m, n = case["m"], case["n"]
        s["a"] = _values(gen, (n, m + case["pad"]))
        s["x"] = _values(gen, (n if case["trans"] == "N" else m,))
        s["y"] = _values(gen, (m if case["trans"] == "N" else n,))
    elif op in ("dot", "axpy"):
        s["x"], s["y"] = _values(gen, (case["n"],)), _values(gen, (case["n"],))
        s["alpha"] = _scalar(rng, 0.5, 2.0)
    elif op == "grouped":
        shapes = _shapes(case)
        for name, count in (("a", lambda m, n, k: m * k), ("b", lambda m, n, k: k * n), ("c", lambda m, n, k: m * n)):
            sizes = [count(*x) for x in shapes]
            s[name] = _values(gen, (sum(sizes),))
            s[name + "_at"] = np.concatenate([[0], np.cumsum(sizes)])[:-1]
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"], op = case, case["op"]
    if op == "gemm_host":
        for name in "abc":
            s[name] = s[name].cpu().numpy()
    elif op == "trsm":
        s["c"] = torch.empty_like(s["b"])   # the solution overwrites a copy of the right-hand sides
    elif op == "grouped":
        shapes = _shapes(case)
        m, n, k = ([x[i] for x in shapes] for i in range(3))
        at = {q: [s[q].data_ptr() + 16 * int(v) for v in s[q + "_at"]] for q in "abc"}
        count = len(shapes)
        s["batch"] = _library()._grouped_arrays(["N"] * count, ["N"] * count, m, n, k, [s["alpha"]] * count, at["a"],
                                                m, at["b"], k, [s["beta"]] * count, at["c"], m)
        s["pointers"] = [x.ctypes.data for x in s["batch"][1:]]
    out = s["c"] if "c" in s else s.get("y")
    if op != "dot":
        s["out"] = {"hi": out[..., 0], "lo": out[..., 1]}
    return s


# ---- one pass --------------------------------------------------------------------------------


def run(s):
    lib, case = _library(), s["case"]
    op = case["op"]
    if op in ("gemm", "gemm_host"):
        lib.mgemm(case["ta"], case["tb"], case["m"], case["n"], case["k"], s["alpha"], s["a"], s["a"].shape[1], s["b"],
                  s["b"].shape[1], s["beta"], s["c"], s["c"].shape[1])
    elif op == "wgemm":
        lib.wgemm(case["ta"], case["tb"], case["m"], case["n"], case["k"], s["alpha"], s["a"], s["a"].shape[1], s["b"],
                  s["b"].shape[1], s["beta"], s["c"], s["c"].shape[1])
    elif op == "syrk":
        lib.msyrk(case["uplo"], case["trans"], case["n"], case["k"], s["alpha"], s["a"], s["a"].shape[1], s["beta"],
                  s["c"], case["n"])
    elif op == "trsm":
        s["c"].copy_(s["b"])
        lib.mtrsm(case["side"], case["uplo"], case["trans"], case["diag"], case["m"], case["n"], s["alpha"], s["a"],
                  s["a"].shape[1], s["c"], case["m"])
    elif op == "gemv":
        lib.mgemv(case["trans"], case["m"], case["n"], s["alpha"], s["a"], s["a"].shape[1], s["x"], 1, s["beta"],
                  s["y"], 1)
    elif op == "dot":
        hi, lo = lib.mdot(case["n"], s["x"], 1, s["y"], 1)
        return {"hi": hi, "lo": lo}
    elif op == "axpy":
        lib.maxpy(case["n"], s["alpha"], s["x"], 1, s["y"], 1)
    elif op == "grouped":
        if lib.lib.mgemm_grouped(s["batch"][0], *s["pointers"]) != 0:
            raise RuntimeError(lib.last_error()[1])
    if lib.last_error()[0] != 0:
        raise RuntimeError(lib.last_error()[1])
    return s["out"]


# ---- the work a call cannot do without -------------------------------------------------------


def work(case):
    """Each operand read once and each output written once; flops are double-double multiplications and additions."""
    op = case["op"]
    if op in ("gemm", "gemm_host", "wgemm"):
        m, n, k, c = case["m"], case["n"], case["k"], 2 if op == "wgemm" else 1
        reads_c = 1 if case.get("beta", True) else 0
        return {"bytes": 16.0 * c * (m * k + k * n + (1 + reads_c) * m * n), "flops": 2.0 * c * c * m * n * k}
    if op == "syrk":
        n, k = case["n"], case["k"]
        return {"bytes": 16.0 * (n * k + n * (n + 1)), "flops": 1.0 * n * (n + 1) * k}
    if op == "trsm":
        m, n = case["m"], case["n"]
        order = m if case["side"] == "L" else n
        return {"bytes": 16.0 * (order * (order + 1) / 2 + 2 * m * n), "flops": 1.0 * m * n * order}
    if op == "gemv":
        m, n = case["m"], case["n"]
        return {"bytes": 16.0 * (m * n + m + n + (m if case["trans"] == "N" else n)), "flops": 2.0 * m * n}
    if op == "grouped":
        shapes = _shapes(case)
        return {"bytes": 16.0 * sum(m * k + k * n + 2 * m * n for m, n, k in shapes),
                "flops": 2.0 * sum(m * n * k for m, n, k in shapes)}
    return {"bytes": (32.0 if op == "dot" else 48.0) * case["n"], "flops": 2.0 * case["n"]}


# ---- the same in plain 64 bits ---------------------------------------------------------------


def exact(case, seed):
    s, op = _inputs(case, seed), case["op"]
    alpha, beta = s["alpha"], s["beta"]
    if op in ("gemm", "gemm_host"):
        a, b, c = (s[q][..., 0] for q in "abc")   # transposes of the matrices, with padding
        m, n, k = case["m"], case["n"], case["k"]
        a = a[:, :m].T if case["ta"] == "N" else a[:, :k]
        b = b[:, :k].T if case["tb"] == "N" else b[:, :n]
        c[:, :m] = (alpha[0] * (a @ b)).T + beta[0] * c[:, :m]
        return {"hi": c, "lo": None}
    if op == "wgemm":
        a, b, c = (torch.complex(s[q][..., 0, 0].contiguous(), s[q][..., 1, 0].contiguous()) for q in "abc")
        a = {"N": lambda v: v.T, "T": lambda v: v, "C": lambda v: v.conj()}[case["ta"]](a)
        b = {"N": lambda v: v.T, "T": lambda v: v, "C": lambda v: v.conj()}[case["tb"]](b)
        c = complex(*alpha[:, 0]) * (a @ b).T + complex(*beta[:, 0]) * c
        return {"hi": torch.view_as_real(c), "lo": None}
    if op == "syrk":
        a, c = s["a"][..., 0], s["c"][..., 0]
        a = a.T if case["trans"] == "N" else a
        full = alpha[0] * (a @ a.T) + beta[0] * c.T   # [row, column]
        keep = torch.ones_like(c, dtype=torch.bool)
        keep = keep.triu() if case["uplo"] == "U" else keep.tril()
        return {"hi": torch.where(keep, full, c.T).T, "lo": None}
    if op == "trsm":
        a, b = s["a"][..., 0].T, alpha[0] * s["b"][..., 0].T
        upper = case["uplo"] == "U"
        a = a.triu() if upper else a.tril()
        if case["trans"] == "T":
            a, upper = a.T, not upper
        x = torch.linalg.solve_triangular(a, b, upper=upper, left=case["side"] == "L",
                                          unitriangular=case["diag"] == "U")
        return {"hi": x.T, "lo": None}
    if op == "gemv":
        a = s["a"][:, :case["m"], 0]
        a = a.T if case["trans"] == "N" else a
        return {"hi": alpha[0] * (a @ s["x"][:, 0]) + beta[0] * s["y"][:, 0], "lo": None}
    if op == "dot":
        # high limbs' product, with what the low limbs add to it
        x, y = s["x"], s["y"]
        return {"hi": float((x[:, 0] * y[:, 0] + (x[:, 0] * y[:, 1] + x[:, 1] * y[:, 0])).sum()), "lo": None}
    if op == "axpy":
        return {"hi": s["y"][:, 0] + alpha[0] * s["x"][:, 0], "lo": None}
    c = s["c"][:, 0]
    for (m, n, k), i, j, l in zip(_shapes(case), s["a_at"], s["b_at"], s["c_at"]):
        a, b = s["a"][i:i + m * k, 0].reshape(k, m), s["b"][j:j + k * n, 0].reshape(n, k)
        at = slice(int(l), int(l) + m * n)
        c[at] = (alpha[0] * (b @ a) + beta[0] * c[at].reshape(n, m)).reshape(-1)
    return {"hi": c, "lo": None}
