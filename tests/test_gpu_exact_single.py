"""Large single-precision products (S, C) through exact INT8 arithmetic: the
product of the operands' integers is exact, so the result is the 64-bit one
rounded once and must be as near to it as the plain FP64 kernel's; operands
that do not fit (a wide spread inside a row, Inf, NaN) run the plain kernel,
bit for bit."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = {"s": (0, np.float32), "c": (2, np.complex64)}
OPS = {"N": lambda x: x, "T": lambda x: x.T, "C": lambda x: x.conj().T}


def mat(r, t, rows, cols):
    v = r.random((rows, cols)) - 0.5
    if t == "c":
        v = v + 1j * (r.random((rows, cols)) - 0.5)
    return np.asfortranarray(v.astype(DT[t][1]))


def call(xk, t, opA, opB, A, B, C0, beta, uplo=0, herm=0, exact=True, pad=0, fits=True,
         count=None):
    """fits: whether the device takes the exact form; count: its moduli."""
    import torch
    code, dt = DT[t]

    def dev(X):
        b = np.zeros((X.shape[1], X.shape[0] + pad), dt)
        b[:, :X.shape[0]] = X.T
        return torch.from_numpy(b).cuda()

    M, N = C0.shape
    K = A.shape[1] if opA == "N" else A.shape[0]
    dA = dev(A)
    dB = dA if B is A else dev(B)
    dC = dev(C0)
    g = xk.GemmArgs(code, "NTC".index(opA), "NTC".index(opB), M, N, K, dA.data_ptr(),
                    A.shape[0] + pad, dB.data_ptr(), B.shape[0] + pad, dC.data_ptr(), M + pad)
    g.alpha[0], g.beta[0] = 0.75, beta
    if t == "c" and not herm:
        g.alpha[1] = -0.5
    g.uplo, g.herm_diag = uplo, herm
    lib = xk.lib()
    lib.xkb_tune_set(b"gemm_exact", 1.0 if exact else 0.0)
    lib.xkb_tune_set(b"gemm_exact_min", 0.0)
    try:
        torch.cuda.synchronize()
        xk.exact_counts(reset=True)
        assert lib.xkb_cuda_gemm(ctypes.byref(g), None) == 0
        xk.sync()
        calls, plain, last = xk.exact_counts()
    finally:
        lib.xkb_tune_set(b"gemm_exact", 1.0)
        lib.xkb_tune_set(b"gemm_exact_min", 3.4e9)
    assert lib.xkb_cuda_take_device_error() == 0
    assert (calls, plain) == ((1, 0 if fits else 1) if exact else (0, 0))
    if exact:
        assert (last > 0) == fits and (count is None or last == count), last
    return np.asfortranarray(dC.cpu().numpy()[:, :M].T)


CASES = [  # (opA, opB, M, N, K, pad, beta, uplo)
    ("N", "N", 512, 512, 512, 0, 0.0, 0),
    ("T", "N", 513, 640, 515, 1, 0.5, 0),
    ("N", "T", 770, 520, 1025, 3, 0.5, 0),
    ("T", "T", 600, 777, 640, 0, 0.0, 0),
    ("N", "T", 700, 700, 600, 0, 0.5, 1),
    ("T", "N", 515, 515, 900, 2, 0.0, 2),
]


@pytest.mark.parametrize("t", "sc")
@pytest.mark.parametrize("case", CASES)
def test_exact_product(xk, t, case):
    opA, opB, M, N, K, pad, beta, uplo = case
    if t == "c":  # conjugated operands too
        opA, opB = opA.replace("T", "C"), opB
    r = np.random.default_rng(M + K)
    A = mat(r, t, *((M, K) if opA == "N" else (K, M)))
    B = mat(r, t, *((K, N) if opB == "N" else (N, K)))
    C0 = mat(r, t, M, N)
    wide = np.complex128 if t == "c" else np.float64
    alpha = 0.75 - 0.5j if t == "c" else 0.75
    ref = alpha * (OPS[opA](A.astype(wide)) @ OPS[opB](B.astype(wide))) + beta * C0
    keep = np.ones((M, N), bool)
    if uplo:
        keep = np.tril(keep) if uplo == 1 else np.triu(keep)
    out = {e: call(xk, t, opA, opB, A, B, C0, beta, uplo, exact=e, pad=pad) for e in (True, False)}
    for e in out:
        assert np.array_equal(out[e][~keep], C0[~keep])
    err = {e: np.linalg.norm((out[e] - ref)[keep]) / np.linalg.norm(ref[keep]) for e in out}
    # both are the 64-bit result rounded once: they differ where that lies
    # within its own 1e-16 of a rounding boundary
    assert err[True] <= 1.001 * err[False], err
    assert np.mean(out[True] != out[False]) < 1e-4


def test_exact_herk_one_buffer(xk):
    """C = A A^H: one set of residue planes serves both operands."""
    r = np.random.default_rng(3)
    A, C0 = mat(r, "c", 600, 530), mat(r, "c", 600, 600)
    C0 = np.asfortranarray((C0 + C0.conj().T).astype(np.complex64))
    w = A.astype(np.complex128)
    keep = np.tril(np.ones((600, 600), bool))
    for opA, opB, X, ref in (("N", "C", A, w @ w.conj().T),):
        out = {e: call(xk, "c", opA, opB, X, X, C0, 0.5, 1, 1, exact=e) for e in (True, False)}
        ref = 0.75 * ref + 0.5 * C0
        err = {e: np.linalg.norm((out[e] - ref)[keep]) / np.linalg.norm(ref[keep]) for e in out}
        assert err[True] <= 1.001 * err[False], err
        assert not out[True].diagonal().imag.any()


@pytest.mark.parametrize("t", "sc")
@pytest.mark.parametrize("what", ["spread", "inf", "nan", "zero", "ints"])
def test_operands_that_do_and_do_not_fit(xk, t, what):
    r = np.random.default_rng(11)
    A, B = mat(r, t, 520, 600), mat(r, t, 600, 540)
    C0 = mat(r, t, 520, 540)
    if what == "spread":  # 90 binary orders inside a row
        A *= np.exp2(r.integers(-45, 46, A.shape)).astype(np.float32)
    elif what == "inf":
        A[3, 5] = np.inf
    elif what == "nan":
        B[7, 9] = np.nan
    elif what == "zero":
        A[5, :] = 0.0
        B[:, 4] = 0.0
    else:
        A = np.asfortranarray(np.round(A * 8))
        B = np.asfortranarray(np.round(B * 8))
    got = call(xk, t, "N", "N", A, B, C0, 0.5, fits=what in ("zero", "ints"))
    plain = call(xk, t, "N", "N", A, B, C0, 0.5, exact=False)
    if what in ("spread", "inf", "nan", "ints"):
        assert np.array_equal(got, plain, equal_nan=True)
    else:
        assert np.allclose(got, plain, rtol=0, atol=1e-5)
        assert np.array_equal(got[5, :], plain[5, :]) and np.array_equal(got[:, 4], plain[:, 4])


# budgets of the scaled operands (bits from a row's lowest set bit up to its
# norm) of the fewest and the most moduli a product may take, and these counts:
# floor((log2 P - 1) / 2) - 1 of the largest pairwise coprime numbers from 256
# down; complex floor((log2 P - 2) / 2) of those whose prime factors are 1 mod 4
BUDGET = {"s": ((30, 8), (57, 15)), "c": ((33, 9), (57, 16))}


@pytest.mark.parametrize("t", "sc")
@pytest.mark.parametrize("end", [0, 1])
def test_moduli_count_at_the_ends_of_its_range(xk, t, end):
    """One entry far below its row's norm asks for exactly the budget of the
    fewest and of the most moduli, then for one bit more: that takes the next
    count, and beyond the most the plain kernel."""
    r = np.random.default_rng(21)
    bits, count = BUDGET[t][end]
    A = np.asfortranarray(r.integers(0, 2, (512, 512)).astype(DT[t][1]))
    B = np.asfortranarray(r.integers(-1, 2, (512, 520)).astype(DT[t][1]))
    A[0, :] = 0
    A[0, 0], A[0, 2] = 1.5, 1  # norm 1.80: exponent 1
    C0 = mat(r, t, 512, 520)
    for more in (0, 1):
        A[0, 1] = 2.0 ** (1 - bits - more)
        fits = end == 0 or more == 0
        got = call(xk, t, "N", "N", A, B, C0, 0.0, fits=fits,
                   count=(count + more) if fits else 0)
        wide = np.complex128 if t == "c" else np.float64
        ref = (0.75 - 0.5j if t == "c" else 0.75) * (A.astype(wide) @ B.astype(wide))
        # sums of at most 512 small integers: exact in 64 bits but for row 0
        assert np.array_equal(got[1:], ref[1:].astype(DT[t][1]))
        assert np.allclose(got[0], ref[0], rtol=2.0 ** -23, atol=0)


@pytest.mark.parametrize("t", "sc")
def test_results_far_below_the_norms_are_exact(xk, t):
    """Rows of 2^-40 to 1 (columns too), and entries whose products lie up to
    2^16 below the norms' product: every result is a small integer times a
    power of two and must come out exactly."""
    r = np.random.default_rng(22)

    def ints(m, n):
        v = r.integers(-4, 5, (m, n)).astype(np.float64)
        return v + 1j * r.integers(-4, 5, (m, n)) if t == "c" else v

    M, N, K = 600, 530, 700
    k = 2.0 ** r.integers(-8, 9, K)
    a = 2.0 ** -r.integers(0, 41, M)[:, None]
    b = 2.0 ** -r.integers(0, 41, N)[None, :]
    iA, iB = ints(M, K), ints(K, N)
    A = np.asfortranarray((a * iA * k[None, :]).astype(DT[t][1]))
    B = np.asfortranarray((b * iB / k[:, None]).astype(DT[t][1]))
    ref = (0.75 - 0.5j if t == "c" else 0.75) * (a * (iA @ iB) * b)
    got = call(xk, t, "N", "N", A, B, np.zeros((M, N), DT[t][1], order="F"), 0.0)
    assert np.array_equal(got, ref.astype(DT[t][1]))
