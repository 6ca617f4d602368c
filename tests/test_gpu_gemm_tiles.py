"""The FP64 tile GEMM at the edges of its two tile shapes, of a stage's k range
and of the vector accesses to C, for every storage type and operand layout,
and its split-K.  The bound is the reference's GEMM bound (checks.gemm_ratio,
3 eps of the storage precision)."""
import ctypes

import numpy as np
import pytest

from tests import checks

pytestmark = pytest.mark.gpu

DT = {"s": (0, np.float32), "d": (1, np.float64), "c": (2, np.complex64),
      "z": (3, np.complex128)}
OPS = {"N": lambda x: x, "T": lambda x: x.T, "C": lambda x: x.conj().T}


def run(xk, t, opA, opB, M, N, K, beta, uplo=0, pad=0, off=0, seed=0):
    import torch
    code, dt = DT[t]
    r = np.random.default_rng(seed)

    def mat(rows, cols):
        v = r.random((rows, cols)) - 0.5
        if t in "cz":
            v = v + 1j * (r.random((rows, cols)) - 0.5)
        return np.asfortranarray(v.astype(dt))

    def dev(X):  # column major, `pad` extra rows, base `off` elements in
        b = np.zeros(off + (X.shape[0] + pad) * X.shape[1], dt)
        v = b[off:].reshape(X.shape[1], X.shape[0] + pad)
        v[:, :X.shape[0]] = X.T
        return torch.from_numpy(b).cuda()

    A = mat(M, K) if opA == "N" else mat(K, M)
    B = mat(K, N) if opB == "N" else mat(N, K)
    C0 = mat(M, N)
    dA, dB, dC = dev(A), dev(B), dev(C0)
    es = np.dtype(dt).itemsize
    g = xk.GemmArgs(code, "NTC".index(opA), "NTC".index(opB), M, N, K, dA.data_ptr() + off * es,
                    A.shape[0] + pad, dB.data_ptr() + off * es, B.shape[0] + pad,
                    dC.data_ptr() + off * es, M + pad)
    alpha = 0.75 - 0.5j if t in "cz" else 0.75
    g.alpha[0], g.alpha[1] = alpha.real, alpha.imag
    g.beta[0] = beta
    g.uplo = uplo
    torch.cuda.synchronize()
    assert xk.lib().xkb_cuda_gemm(ctypes.byref(g), None) == 0
    xk.sync()
    out = dC.cpu().numpy()
    assert xk.lib().xkb_cuda_take_device_error() == 0
    full = out[off:].reshape(N, M + pad)
    assert not full[:, M:].any()  # the padding rows are not written
    C = np.asfortranarray(full[:, :M].T)
    wide = np.complex128 if t in "cz" else np.float64
    ref = alpha * (OPS[opA](A.astype(wide)) @ OPS[opB](B.astype(wide))) + beta * C0
    if uplo:
        keep = np.tril(np.ones((M, N), bool)) if uplo == 1 else np.triu(np.ones((M, N), bool))
        assert np.array_equal(C[~keep], C0[~keep])
        ref = np.where(keep, ref, C0)
    assert checks.gemm_ratio(C, ref, A, B, C0, alpha, beta, K) <= 3.0


@pytest.mark.parametrize("t", "sdcz")
@pytest.mark.parametrize("tile", [0.0, 1e9])  # 64 x 64 always, 32 x 32 always (real types)
def test_tile_edges(xk, t, tile):
    lib = xk.lib()
    lib.xkb_tune_set(b"gemm_tile64_min_blocks", tile)
    try:
        ops = "NT" if t in "sd" else "NTC"
        seed = 0
        for opA in ops:
            for opB in ops:
                for M, N, K, pad, off in ((1, 1, 1, 0, 0), (31, 33, 7, 1, 0), (32, 32, 8, 0, 0),
                                          (33, 64, 17, 0, 1), (64, 65, 32, 3, 0),
                                          (65, 31, 33, 0, 0), (130, 97, 66, 2, 0),
                                          (2, 200, 129, 0, 0)):
                    seed += 1
                    run(xk, t, opA, opB, M, N, K, 0.5 * (seed % 2), pad=pad, off=off, seed=seed)
    finally:
        lib.xkb_tune_set(b"gemm_tile64_min_blocks", -1.0)


@pytest.mark.parametrize("t", "sdcz")
@pytest.mark.parametrize("uplo", [1, 2])
def test_masked_edges(xk, t, uplo):
    for i, (M, N, K) in enumerate(((63, 63, 16), (64, 64, 9), (97, 97, 40), (130, 130, 31))):
        run(xk, t, "N", "T", M, N, K, 0.5, uplo=uplo, pad=i % 3, seed=10 + i)


@pytest.mark.parametrize("t", "sdcz")
def test_split_k_edges(xk, t):
    """Few tiles and a long, odd K: the slices and their reduction."""
    for i, (M, N, K, uplo) in enumerate(((33, 31, 4097, 0), (100, 40, 3001, 0),
                                         (65, 65, 2050, 1))):
        run(xk, t, "T" if i % 2 else "N", "N", M, N, K, 0.5, uplo=uplo, pad=i, seed=20 + i)
