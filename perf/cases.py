"""Performance cases of the library, each one pass through its public entry
points (the C ABI of include/xkblas.h and include/xkb_cuda.h).

listed() names twelve calls that programs make of a level-3 BLAS with a
tensor-op mode, a batch executor and tile factorizations, from the smallest
calls to the largest; draw() gives further calls of the same ranges.  Inputs
are what the library's tests and benchmark use: entries uniform in
[-0.5, 0.5], triangles and factorized matrices with a dominant diagonal, and
for the wide-spread contraction exponents in [-20, 20] per row of A and per
column of B.  Matrices are column major; a buffer is kept as a (columns, ld)
torch tensor, so buf[:, :rows].t() is the matrix.
"""
import ctypes
import math

import numpy as np
import torch

import xkblas_b200 as X

DT = {"s": 0, "d": 1, "c": 2, "z": 3}
TORCH = {"s": torch.float32, "d": torch.float64, "c": torch.complex64, "z": torch.complex128}
NUMPY = {"s": np.float32, "d": np.float64, "c": np.complex64, "z": np.complex128}
ES = {"s": 4, "d": 8, "c": 8, "z": 16}
OP = {"N": 0, "T": 1, "C": 2}
CBLAS_OP = {"N": 111, "T": 112, "C": 113}
CBLAS_UPLO = {"L": 122, "U": 121}
FULL, LOWER, UPPER = 0, 1, 2
UPLO = {"L": LOWER, "U": UPPER}
OZAKI_MIN = 2048  # the library's default crossover of the tensor-op mode
_stream = None


def listed():
    return [
        # the smallest calls: one contraction of a blocked algorithm's inner
        # block, called in a loop (latency and launches count)
        dict(name="dgemm small", kind="gemm", t="d", opA="N", opB="N", M=96, N=80, K=64, ld=0,
             alpha=1.0, beta=1.0),
        # the benchmark's plain FP64 configuration
        dict(name="dgemm 1024", kind="gemm", t="d", opA="N", opB="N", M=1024, N=1024, K=1024,
             ld=0, alpha=1.5, beta=-0.5),
        # a tall product of a sub-matrix view: odd sizes, odd leading
        # dimensions, op(A) transposed
        dict(name="dgemm ragged", kind="gemm", t="d", opA="T", opB="N", M=3001, N=517, K=777,
             ld=3, alpha=1.0, beta=0.0),
        # complex double, conjugated operand (the mixed batch's type at an
        # ordinary size)
        dict(name="zgemm", kind="gemm", t="z", opA="N", opB="C", M=1200, N=900, K=1100, ld=0,
             alpha=1.0, beta=0.5),
        # single precision at an ordinary large size
        dict(name="sgemm 4096", kind="gemm", t="s", opA="N", opB="T", M=4096, N=4096, K=4096,
             ld=0, alpha=1.0, beta=0.0),
        # tensor-op mode, ordinary size
        dict(name="dgemm tensor-op 4096", kind="oz", t="d", opA="N", opB="N", M=4096, N=4096,
             K=4096, ld=0, spread=0, alpha=1.0, beta=0.5),
        # tensor-op mode, the headline: wide exponent spread, the largest call
        dict(name="dgemm tensor-op 16384", kind="oz", t="d", opA="N", opB="N", M=16384, N=16384,
             K=16384, ld=0, spread=20, alpha=1.0, beta=0.0),
        # complex Hermitian rank-k update in tensor-op mode (benchmark shape)
        dict(name="zherk tensor-op 8192", kind="rk", t="z", uplo="L", trans="N", N=8192, K=8192,
             ld=0, tc=1),
        # the benchmark's triangular solve
        dict(name="dtrsm 4096", kind="trsm", t="d", side="L", uplo="L", trans="N", diag=0, M=4096,
             N=4096, ld=0, tc=0),
        # Cholesky factorization, plain FP64
        dict(name="dpotrf 8192", kind="potrf", t="d", uplo="L", N=8192, ld=0, tc=0),
        # a stream of uneven calls as one batch (the benchmark's mix)
        dict(name="batch 300 mixed", kind="batch", calls=300, mix=1),
        # the public synchronous call on host matrices: upload, product, copy back
        dict(name="dgemm host 2048", kind="host", t="d", call="gemm", M=2048, N=2048, K=2048),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "gemm", "oz", "oz", "rk", "trsm", "trsm", "trmm", "symm",
                       "potrf", "getrf", "batch", "host"])
    ld = rng.choice([0, 0, 1, 3, 8])
    if kind == "gemm":
        t = rng.choice("dddzzsscc")
        top = 4096 if t in "sd" else 2400
        ops = "NT" if t in "sd" else "NTC"
        return dict(kind=kind, t=t, opA=rng.choice(ops), opB=rng.choice(ops),
                    M=_log(rng, 48, top), N=_log(rng, 48, top), K=_log(rng, 48, top), ld=ld,
                    alpha=1.0, beta=rng.choice([0.0, 0.5]))
    if kind == "oz":
        t = rng.choice("dddz")
        top = 8192 if t == "d" else 5000
        return dict(kind=kind, t=t, opA=rng.choice("NT"), opB=rng.choice("NT"),
                    M=_log(rng, 2048, top), N=_log(rng, 2048, top), K=_log(rng, 2048, top), ld=ld,
                    spread=rng.choice([0, 20]), alpha=1.0, beta=rng.choice([0.0, 0.5]))
    if kind == "rk":
        tc = rng.choice([0, 1])
        t = rng.choice("dz") if tc else rng.choice("sddzz")
        lo, hi = (2048, 6144) if tc else (200, 3000)
        return dict(kind=kind, t=t, uplo=rng.choice("LU"),
                    trans=rng.choice("NC" if t == "z" else "NT"), N=_log(rng, lo, hi),
                    K=_log(rng, lo, hi), ld=ld, tc=tc)
    if kind == "trsm":
        tc = rng.choice([0, 0, 1])
        t = rng.choice("dddzs") if not tc else "d"
        side = rng.choice("LR")
        n, m = _log(rng, 128, 6144 if t == "d" else 3000), _log(rng, 64, 4096)
        return dict(kind=kind, t=t, side=side, uplo=rng.choice("LU"),
                    trans=rng.choice("NTC" if t == "z" else "NT"), diag=rng.choice([0, 0, 1]),
                    M=n if side == "L" else m, N=m if side == "L" else n, ld=ld, tc=tc)
    if kind == "trmm":
        side = rng.choice("LR")
        return dict(kind=kind, t=rng.choice("ddzs"), side=side, uplo=rng.choice("LU"),
                    trans=rng.choice("NT"), diag=rng.choice([0, 1]), M=_log(rng, 200, 3000),
                    N=_log(rng, 200, 3000), ld=ld, tc=0)
    if kind == "symm":
        return dict(kind=kind, t=rng.choice("ddzs"), side=rng.choice("LR"), uplo=rng.choice("LU"),
                    M=_log(rng, 200, 3000), N=_log(rng, 200, 3000), ld=ld, tc=0)
    if kind in ("potrf", "getrf"):
        t = rng.choice("dddzs")
        d = dict(kind=kind, t=t, N=_log(rng, 200, 8192 if t == "d" else 4000), ld=ld,
                 tc=rng.choice([0, 1]) if t == "d" else 0)
        if kind == "potrf":
            d["uplo"] = rng.choice("LU")
        return d
    if kind == "batch":
        return dict(kind=kind, calls=_log(rng, 16, 400), mix=rng.randrange(2, 1 << 20))
    return dict(kind="host", t=rng.choice("ddz"), call=rng.choice(["gemm", "gemm", "trsm"]),
                M=_log(rng, 100, 2600), N=_log(rng, 100, 2600), K=_log(rng, 100, 2600))


# ---- inputs -----------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _mat(g, t, rows, cols, pad):
    """A (cols, rows + pad) buffer of uniform [-0.5, 0.5] entries (per part)."""
    wide = torch.complex128 if t in "cz" else torch.float64
    shape = (cols, rows + pad)
    if t in "cz":
        v = torch.view_as_complex(torch.rand(shape + (2,), generator=g, device="cuda",
                                             dtype=torch.float64).sub_(0.5))
    else:
        v = torch.rand(shape, generator=g, device="cuda", dtype=wide).sub_(0.5)
    return v.to(TORCH[t])


def _dominant(buf, n, add):
    """Adds `add` to the diagonal of the n x n matrix in the buffer."""
    buf[:, :n].diagonal().add_(add)
    return buf


def _pair(re, im=0.0):
    return (ctypes.c_double * 2)(re, im)


def _dptr(p):
    return ctypes.cast(p, ctypes.POINTER(ctypes.c_double))


def _sp():
    global _stream
    X.init()
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream, ctypes.c_void_p(_stream.cuda_stream)


def _gemm_args(t, opA, opB, M, N, K, A, B, C, alpha, beta, uplo=FULL, herm=0):
    a = X.GemmArgs(DT[t], OP[opA], OP[opB], M, N, K, A.data_ptr(), A.shape[1], B.data_ptr(),
                   B.shape[1], C.data_ptr(), C.shape[1])
    a.alpha[0], a.beta[0] = alpha, beta
    a.uplo, a.herm_diag = uplo, herm
    return a


def _shape(op, r, c):
    return (r, c) if op == "N" else (c, r)


def _spread(case, g, rows, cols, along_rows):
    """Exponents uniform in [-spread, spread] per row (or column)."""
    n = rows if along_rows else cols
    e = torch.randint(-case["spread"], case["spread"] + 1, (n,), generator=g, device="cuda")
    return torch.pow(2.0, e.to(torch.float64))


def prepare(case, seed):
    stream, sp = _sp()
    lib = X.lib()
    g = _gen(seed)
    k = case["kind"]
    s = {"case": case, "lib": lib, "sp": sp, "stream": stream}
    if k in ("gemm", "oz"):
        t, M, N, K, pad = case["t"], case["M"], case["N"], case["K"], case["ld"]
        s["A"] = _mat(g, t, *_shape(case["opA"], M, K), pad)
        s["B"] = _mat(g, t, *_shape(case["opB"], K, N), pad)
        s["C"] = _mat(g, t, M, N, pad)
        if case.get("spread"):
            # exponents per row of op(A) and per column of op(B)
            ea, eb = _spread(case, g, M, K, True), _spread(case, g, K, N, False)
            ra, rb = _shape(case["opA"], M, K)[0], _shape(case["opB"], K, N)[0]
            s["A"][:, :ra] *= ea[None, :] if case["opA"] == "N" else ea[:, None]
            s["B"][:, :rb] *= eb[:, None] if case["opB"] == "N" else eb[None, :]
        s["args"] = _gemm_args(t, case["opA"], case["opB"], M, N, K, s["A"], s["B"], s["C"],
                               case["alpha"], case["beta"])
        s["ref"] = ctypes.byref(s["args"])
    elif k == "rk":
        t, N, K, pad = case["t"], case["N"], case["K"], case["ld"]
        herm = t == "z"
        s["A"] = _mat(g, t, *_shape(case["trans"], N, K), pad)
        s["C"] = _mat(g, t, N, N, pad)
        v = s["C"][:, :N]
        v.copy_(0.5 * (v + (v.mH if herm else v.mT)))
        tr = "C" if herm else "T"
        opA, opB = ("N", tr) if case["trans"] == "N" else (tr, "N")
        s["args"] = _gemm_args(t, opA, opB, N, N, K, s["A"], s["A"], s["C"], 1.0, 0.5,
                               UPLO[case["uplo"]], 1 if herm else 0)
        s["ref"] = ctypes.byref(s["args"])
    elif k in ("trsm", "trmm", "symm"):
        t, M, N, pad = case["t"], case["M"], case["N"], case["ld"]
        n = M if case["side"] == "L" else N
        s["A"] = _mat(g, t, n, n, pad)
        if k == "trsm":
            if case["diag"]:
                s["A"] /= n  # unit diagonal: a well-conditioned triangle
            else:
                _dominant(s["A"], n, n)
        s["B0"] = _mat(g, t, M, N, pad)
        s["al"] = _pair(2.0 if k == "trsm" else 1.0)
        s["be"] = _pair(0.5)
        oz = OZAKI_MIN if case["tc"] else 0
        side = 0 if case["side"] == "L" else 1
        if k == "symm":
            s["C"] = _mat(g, t, M, N, pad)
            s["argv"] = (DT[t], 0, side, UPLO[case["uplo"]], M, N, _dptr(s["al"]),
                         s["A"].data_ptr(), s["A"].shape[1], s["B0"].data_ptr(),
                         s["B0"].shape[1], _dptr(s["be"]), s["C"].data_ptr(), s["C"].shape[1], oz,
                         sp)
        else:
            s["B"] = s["B0"].clone()
            s["argv"] = (DT[t], side, UPLO[case["uplo"]], OP[case["trans"]], case["diag"], M, N,
                         _dptr(s["al"]), s["A"].data_ptr(), s["A"].shape[1], s["B"].data_ptr(),
                         s["B"].shape[1], oz, sp)
    elif k in ("potrf", "getrf"):
        t, N, pad = case["t"], case["N"], case["ld"]
        s["A0"] = _mat(g, t, N, N, pad)
        if k == "potrf":
            v = s["A0"][:, :N]
            v.copy_(0.5 * (v + (v.mH if t in "cz" else v.mT)))
        _dominant(s["A0"], N, N)
        s["A"] = s["A0"].clone()
        s["info"] = torch.zeros(1, dtype=torch.int32, device="cuda")
        oz = OZAKI_MIN if case["tc"] else 0
        head = (DT[t], UPLO[case["uplo"]], N) if k == "potrf" else (DT[t], N)
        s["argv"] = head + (s["A"].data_ptr(), s["A"].shape[1], s["info"].data_ptr(), oz, sp)
    elif k == "batch":
        s.update(_batch(case, g))
    else:
        s.update(_host(case, seed))
    torch.cuda.synchronize()
    return s


def _batch_shapes(case):
    """The mix of the benchmark's batch: 70 % DGEMM, 20 % left lower DTRSM,
    10 % ZGEMM, M, N, K log-uniform in [64, 2048]."""
    r = np.random.default_rng(case["mix"])

    def lu():
        return int(round(math.exp(r.uniform(math.log(64), math.log(2048)))))

    out = []
    for _ in range(case["calls"]):
        x = r.random()
        what = "d" if x < 0.7 else ("trsm" if x < 0.9 else "z")
        out.append((what, lu(), lu(), lu()))
    return out


def _batch(case, g):
    """All operands in three flat buffers per type: read-only, gemm outputs,
    and the triangular solves' right-hand sides (solved in place)."""
    shapes = _batch_shapes(case)
    need = {"d": 0, "z": 0, "C": 0, "Z": 0, "x": 0}
    for what, m, n, k in shapes:
        if what == "trsm":
            need["d"] += m * m + 1
            need["x"] += m * n + 1
        else:
            need[what] += m * k + k * n + 2
            need["C" if what == "d" else "Z"] += m * n + 1
    flat = {"d": _mat(g, "d", need["d"] + 2, 1, 0)[0], "z": _mat(g, "z", need["z"] + 2, 1, 0)[0],
            "C": _mat(g, "d", need["C"] + 2, 1, 0)[0], "Z": _mat(g, "z", need["Z"] + 2, 1, 0)[0],
            "x": _mat(g, "d", need["x"] + 2, 1, 0)[0]}
    at = dict.fromkeys(flat, 0)

    def take(key, rows, cols):
        b = flat[key][at[key]:at[key] + rows * cols]
        at[key] += rows * cols
        if key in "dCx" and at[key] % 2:
            at[key] += 1  # 16-byte aligned bases, as an allocator gives
        return b

    ops, parts = [], []
    for what, m, n, k in shapes:
        o = X.BatchOp()
        if what == "trsm":
            A, B = take("d", m, m), take("x", m, n)
            A.view(m, m).diagonal().add_(m)
            o.kind, o.dtype, o.uplo, o.M, o.N = 1, 1, LOWER, m, n
            o.A, o.lda, o.C, o.ldc = A.data_ptr(), m, B.data_ptr(), m
            o.alpha[0] = 2.0
            parts.append((what, m, n, k, A, B, None))
        else:
            A, B = take(what, m, k), take(what, k, n)
            C = take("C" if what == "d" else "Z", m, n)
            o.kind, o.dtype, o.M, o.N, o.K = 0, DT[what], m, n, k
            o.A, o.lda, o.B, o.ldb, o.C, o.ldc = (A.data_ptr(), m, B.data_ptr(), k, C.data_ptr(),
                                                  m)
            o.alpha[0], o.beta[0] = 1.0, 0.5
            parts.append((what, m, n, k, A, B, C))
        ops.append(o)
    return {"flat": flat, "x0": flat["x"].clone(), "parts": parts, "n": len(ops),
            "ops": (X.BatchOp * len(ops))(*ops)}


def _host(case, seed):
    """Pinned host matrices (xkblas_malloc), as a user of the public API has."""
    t, M, N, K = case["t"], case["M"], case["N"], case["K"]
    r = np.random.default_rng(seed)

    def mat(rows, cols):
        a = X.pinned_empty((rows, cols), NUMPY[t])
        v = r.random((cols, rows)) - 0.5
        a[...] = (v + 1j * (r.random((cols, rows)) - 0.5)).T if t in "cz" else v.T
        return a

    s = {"alpha": np.array([1.5], NUMPY[t]), "beta": np.array([-0.5], NUMPY[t])}
    if case["call"] == "gemm":
        s["A"], s["B"], s["C"] = mat(M, K), mat(K, N), mat(M, N)
        s["argv"] = (111, 111, M, N, K, X._ptr(s["alpha"]), X._ptr(s["A"]), M, X._ptr(s["B"]), K,
                     X._ptr(s["beta"]), X._ptr(s["C"]), M)
        s["f"] = getattr(X.lib(), "xkblas_%sgemm_sync" % t)
    else:
        s["A"], s["B0"], s["B"] = mat(M, M), mat(M, N), mat(M, N)
        s["A"][np.arange(M), np.arange(M)] += M
        s["argv"] = (141, 122, 111, 131, M, N, X._ptr(s["alpha"]), X._ptr(s["A"]), M,
                     X._ptr(s["B"]), M)
        s["f"] = getattr(X.lib(), "xkblas_%strsm_sync" % t)
    return s


# ---- one pass -----------------------------------------------------------------
def _ok(rc):
    if rc != 0:
        raise RuntimeError("the call returned %d" % rc)


def _view(buf, rows):
    return buf[:, :rows].t()


def run(s):
    case, lib = s["case"], s["lib"]
    k = case["kind"]
    if k == "gemm":
        _ok(lib.xkb_cuda_gemm(s["ref"], s["sp"]))
        return _view(s["C"], case["M"])
    if k == "oz":
        _ok(lib.xkb_cuda_ozaki_gemm(s["ref"], 0, s["sp"]))
        return _view(s["C"], case["M"])
    if k == "rk":
        _ok(lib.xkb_cuda_ozaki_gemm(s["ref"], 0, s["sp"]) if case["tc"]
            else lib.xkb_cuda_gemm(s["ref"], s["sp"]))
        return _view(s["C"], case["N"])
    if k in ("trsm", "trmm"):
        with torch.cuda.stream(s["stream"]):
            s["B"].copy_(s["B0"])
        _ok((lib.xkb_cuda_trsm if k == "trsm" else lib.xkb_cuda_trmm)(*s["argv"]))
        return _view(s["B"], case["M"])
    if k == "symm":
        _ok(lib.xkb_cuda_symm(*s["argv"]))
        return _view(s["C"], case["M"])
    if k in ("potrf", "getrf"):
        with torch.cuda.stream(s["stream"]):
            s["A"].copy_(s["A0"])
        _ok((lib.xkb_cuda_potrf if k == "potrf" else lib.xkb_cuda_getrf_nopiv)(*s["argv"]))
        return {"factor": _view(s["A"], case["N"]), "info": s["info"]}
    if k == "batch":
        with torch.cuda.stream(s["stream"]):
            s["flat"]["x"].copy_(s["x0"])
        _ok(lib.xkb_cuda_batch(s["ops"], s["n"], 0, s["sp"]))
        return {"dgemm": s["flat"]["C"], "zgemm": s["flat"]["Z"], "dtrsm": s["flat"]["x"]}
    if case["call"] == "trsm":
        s["B"][...] = s["B0"]
    _ok(s["f"](*s["argv"]))
    return s["C"] if case["call"] == "gemm" else s["B"]


# ---- what a pass cannot do without ----------------------------------------------
def work(case):
    k = case["kind"]
    if k == "batch":
        b = f = 0
        for what, m, n, kk in _batch_shapes(case):
            if what == "trsm":
                b += 8 * (m * (m + 1) // 2 + 2 * m * n)
                f += m * m * n
            else:
                z = 2 if what == "z" else 1
                b += 8 * z * (m * kk + kk * n + 2 * m * n)
                f += (8 if what == "z" else 2) * m * n * kk
        return {"bytes": b, "flops": f}
    t = case["t"]
    es, c = ES[t], 4 if t in "cz" else 1
    if k == "host":
        M, N, K = case["M"], case["N"], case["K"]
        if case["call"] == "gemm":
            return {"bytes": es * (M * K + K * N + 2 * M * N), "flops": 2 * c * M * N * K}
        return {"bytes": es * (M * (M + 1) // 2 + 2 * M * N), "flops": c * M * M * N}
    if k in ("gemm", "oz"):
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": es * (M * K + K * N + M * N * (2 if case["beta"] else 1)),
                "flops": 2 * c * M * N * K}
    if k == "rk":
        N, K = case["N"], case["K"]
        return {"bytes": es * (N * K + N * (N + 1)), "flops": c * N * (N + 1) * K}
    if k in ("trsm", "trmm", "symm"):
        M, N = case["M"], case["N"]
        n = M if case["side"] == "L" else N
        fl = c * n * M * N * (2 if k == "symm" else 1)
        return {"bytes": es * (n * (n + 1) // 2 + (3 if k == "symm" else 2) * M * N), "flops": fl}
    N = case["N"]
    if k == "potrf":
        return {"bytes": es * N * (N + 1), "flops": c * N ** 3 // 3}
    return {"bytes": es * 2 * N * N, "flops": c * 2 * N ** 3 // 3}


# ---- the same results in 64 bits, without the library ----------------------------
def _wide(x):
    return x.to(torch.complex128 if x.is_complex() else torch.float64)


def _op(m, op):
    return m if op == "N" else (m.mT if op == "T" else m.mH)


def _tri(a, uplo, unit=False):
    m = torch.tril(a) if uplo == "L" else torch.triu(a)
    if unit:
        m = m.clone()
        m.diagonal().fill_(1.0)
    return m


def exact(case, seed):
    s = prepare(case, seed)
    k = case["kind"]
    if k in ("gemm", "oz"):
        ra, rb = _shape(case["opA"], case["M"], case["K"])[0], _shape(case["opB"], case["K"],
                                                                      case["N"])[0]
        A, B = _wide(_view(s["A"], ra)), _wide(_view(s["B"], rb))
        out = torch.matmul(_op(A, case["opA"]), _op(B, case["opB"])).mul_(case["alpha"])
        if case["beta"]:
            out += case["beta"] * _wide(_view(s["C"], case["M"]))
        return out
    if k == "rk":
        N, herm = case["N"], case["t"] == "z"
        A = _wide(_view(s["A"], _shape(case["trans"], N, case["K"])[0]))
        if case["trans"] != "N":
            A = _op(A, "C" if herm else "T")
        C = _wide(_view(s["C"], N))
        new = torch.matmul(A, A.mH if herm else A.mT) + 0.5 * C
        if herm:
            new.diagonal().copy_(new.diagonal().real.to(new.dtype))
        keep = torch.ones(N, N, dtype=torch.bool, device=C.device)
        keep = keep.triu(1) if case["uplo"] == "L" else keep.tril(-1)
        return torch.where(keep, C, new)
    if k in ("trsm", "trmm", "symm"):
        M = case["M"]
        n = M if case["side"] == "L" else case["N"]
        A, B = _wide(_view(s["A"], n)), _wide(_view(s["B0"], M))
        if k == "symm":
            T = _tri(A, case["uplo"])
            S = T + T.mT
            S.diagonal().copy_(A.diagonal())
            out = torch.matmul(S, B) if case["side"] == "L" else torch.matmul(B, S)
            return out + 0.5 * _wide(_view(s["C"], M))
        T = _op(_tri(A, case["uplo"], bool(case["diag"])), case["trans"])
        if k == "trmm":
            return torch.matmul(T, B) if case["side"] == "L" else torch.matmul(B, T)
        upper = (case["uplo"] == "U") == (case["trans"] == "N")
        return 2.0 * torch.linalg.solve_triangular(T, B, upper=upper, left=case["side"] == "L",
                                                   unitriangular=bool(case["diag"]))
    if k == "potrf":
        A = _wide(_view(s["A0"], case["N"]))
        L = torch.linalg.cholesky(A if case["uplo"] == "L" else A.mH)
        f = L + torch.triu(A, 1) if case["uplo"] == "L" else L.mH + torch.tril(A, -1)
        return {"factor": f, "info": None}
    if k == "getrf":
        A = _wide(_view(s["A0"], case["N"]))
        return {"factor": torch.linalg.lu_factor(A, pivot=False)[0], "info": None}
    if k == "batch":
        flat = s["flat"]
        out = {"dgemm": flat["C"].clone(), "zgemm": flat["Z"].clone(), "dtrsm": flat["x"].clone()}
        base = {"d": ("dgemm", "C"), "z": ("zgemm", "Z"), "trsm": ("dtrsm", "x")}
        for what, m, n, kk, A, B, C in s["parts"]:
            name, key = base[what]
            res = B if what == "trsm" else C
            off = (res.data_ptr() - flat[key].data_ptr()) // flat[key].element_size()
            if what == "trsm":
                L = torch.tril(A.view(m, m).t())
                new = 2.0 * torch.linalg.solve_triangular(L, B.view(n, m).t(), upper=False)
            else:
                new = A.view(kk, m).t() @ B.view(n, kk).t() + 0.5 * C.view(n, m).t()
            out[name][off:off + m * n] = new.t().reshape(-1)
        return out
    A = torch.from_numpy(np.array(s["A"])).cuda()
    if case["call"] == "gemm":
        B, C = (torch.from_numpy(np.array(s[x])).cuda() for x in "BC")
        return (1.5 * (A @ B) - 0.5 * C).cpu().numpy()
    B = torch.from_numpy(np.array(s["B0"])).cuda()
    return (1.5 * torch.linalg.solve_triangular(torch.tril(A), B, upper=False)).cpu().numpy()
