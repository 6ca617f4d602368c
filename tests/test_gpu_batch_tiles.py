"""The tile-task executor at the edges of its tiles and solve blocks: sizes
around 32 and 64, odd leading dimensions (8-byte staging) and bases that are
not 16-byte aligned, every op and triangle, solves of several blocks whose
later blocks read rows other blocks solved in the same launch."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def dev(X, pad, off):
    import torch
    b = np.zeros(off + (X.shape[0] + pad) * X.shape[1], X.dtype)
    b[off:].reshape(X.shape[1], X.shape[0] + pad)[:, :X.shape[0]] = X.T
    return torch.from_numpy(b).cuda()


def host(d, shape, pad, off):
    return d.cpu().numpy()[off:].reshape(shape[1], shape[0] + pad)[:, :shape[0]].T


def rnd(r, m, n, cplx):
    v = r.random((m, n)) - 0.5
    return v + 1j * (r.random((m, n)) - 0.5) if cplx else v


OPF = [lambda x: x, lambda x: x.T, lambda x: x.conj().T]


@pytest.mark.parametrize("pad,off", [(0, 0), (1, 0), (3, 1)])
@pytest.mark.parametrize("cplx", [False, True])
def test_batch_tile_edges(xk, cplx, pad, off):
    r = np.random.default_rng(7 + pad + off)
    t = 3 if cplx else 1
    es = 16 if cplx else 8
    ops, keep = [], []
    nop = 3 if cplx else 2
    sizes = [(1, 1, 1), (31, 33, 7), (32, 64, 8), (65, 63, 17), (64, 64, 64), (130, 97, 129)]
    for k, (M, N, K) in enumerate(sizes):
        oa, ob = k % nop, (k // nop + k) % nop
        A = rnd(r, *((M, K) if oa == 0 else (K, M)), cplx)
        B = rnd(r, *((K, N) if ob == 0 else (N, K)), cplx)
        C = rnd(r, M, N, cplx)
        d = [dev(X, pad, off) for X in (A, B, C)]
        o = xk.BatchOp()
        o.kind, o.dtype, o.opA, o.opB, o.M, o.N, o.K = 0, t, oa, ob, M, N, K
        o.A, o.lda = d[0].data_ptr() + off * es, A.shape[0] + pad
        o.B, o.ldb = d[1].data_ptr() + off * es, B.shape[0] + pad
        o.C, o.ldc = d[2].data_ptr() + off * es, M + pad
        o.alpha[0], o.beta[0] = 0.75, 0.5
        if cplx:
            o.alpha[1] = -0.25
        al = 0.75 - 0.25j if cplx else 0.75
        ops.append(o)
        ref = al * (OPF[oa](A) @ OPF[ob](B)) + 0.5 * C
        # |C - ref| <= (K + 2) eps (|alpha| |A||B| + |beta||C|), complex twice
        bound = (2 if cplx else 1) * 2 * (K + 4) * EPS * (
            abs(al) * (np.abs(OPF[oa](A)) @ np.abs(OPF[ob](B))) + np.abs(C))
        keep.append((d, (M, N), ref, bound))
    for k, (M, N) in enumerate([(1, 1), (63, 5), (64, 64), (65, 66), (129, 31), (200, 70),
                                (300, 33)]):
        for uplo in (1, 2):
            tr, unit = (k + uplo) % nop, k % 2
            # unit: small off-diagonal entries, else a dominant diagonal
            A = rnd(r, M, M, cplx) / M + np.eye(M)
            B = rnd(r, M, N, cplx)
            d = [dev(A, pad, off), dev(B, pad, off)]
            o = xk.BatchOp()
            o.kind, o.dtype, o.uplo, o.trans, o.diag, o.M, o.N = 1, t, uplo, tr, unit, M, N
            o.A, o.lda = d[0].data_ptr() + off * es, M + pad
            o.C, o.ldc = d[1].data_ptr() + off * es, M + pad
            o.alpha[0] = 2.0
            ops.append(o)
            T = np.tril(A) if uplo == 1 else np.triu(A)
            if unit:
                np.fill_diagonal(T, 1.0)
            T = OPF[tr](T)
            keep.append((d, (M, N), T, B))
    import torch
    arr = (xk.BatchOp * len(ops))(*ops)
    torch.cuda.synchronize()
    assert xk.lib().xkb_cuda_batch(arr, len(ops), 0, None) == 0
    xk.sync()
    assert xk.lib().xkb_cuda_take_device_error() == 0
    for d, shape, ref, bound in keep:
        X = host(d[-1], shape, pad, off)
        if len(d) == 3:
            assert (np.abs(X - ref) <= bound).all(), shape
        else:  # residual: |T X - 2 B| <= c M eps (|T||X| + 2|B|)
            T, B = ref, bound
            lim = 8 * (shape[0] + 4) * EPS * (np.abs(T) @ np.abs(X) + 2 * np.abs(B))
            assert (np.abs(T @ X - 2 * B) <= lim).all(), shape


def solve_batch(xk, T, B, uplo, tr, unit):
    """op(T) X = B by one batch of one call."""
    import torch
    M, N = B.shape
    cplx = np.iscomplexobj(B)
    dT, dB = dev(T, 0, 0), dev(B, 0, 0)
    o = xk.BatchOp()
    o.kind, o.dtype, o.uplo, o.trans, o.diag, o.M, o.N = 1, 3 if cplx else 1, uplo, tr, unit, M, N
    o.A, o.lda, o.C, o.ldc = dT.data_ptr(), M, dB.data_ptr(), M
    o.alpha[0] = 1.0
    torch.cuda.synchronize()
    assert xk.lib().xkb_cuda_batch(ctypes.byref(o), 1, 0, None) == 0
    xk.sync()
    assert xk.lib().xkb_cuda_take_device_error() == 0
    return host(dB, B.shape, 0, 0)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("uplo,tr,unit", [(1, 0, 0), (2, 0, 0), (1, 1, 1), (2, 1, 0)])
def test_nonfinite_right_hand_sides(xk, cplx, uplo, tr, unit):
    """Inf and NaN in a right-hand side reach the unknowns that depend on
    them and no others: those solved earlier, and the other columns, are what
    they are without them."""
    r = np.random.default_rng(4)
    for M in (5, 20, 64, 75):
        A = rnd(r, M, M, cplx) / M + np.eye(M)
        B = rnd(r, M, 19, cplx)
        clean = solve_batch(xk, A, B, uplo, tr, unit)
        bad = B.copy()
        at = {1: (3, np.nan), 4: (M - 2, np.inf), 17: (M // 2, -np.inf), 18: (0, np.nan)}
        for c, (i, v) in at.items():
            bad[i, c] = v
        X = solve_batch(xk, A, bad, uplo, tr, unit)
        fwd = (uplo == 1) == (tr == 0)
        for c in range(19):
            i = at[c][0] if c in at else None
            # unknowns solved before unknown i
            free = slice(0, M) if i is None else (slice(0, i) if fwd else slice(i + 1, M))
            assert np.allclose(X[free, c], clean[free, c], rtol=0, atol=1e-13), (M, c)
            if i is not None:
                assert not np.isfinite(X[i, c]), (M, c)
                dep = X[i:, c] if fwd else X[:i + 1, c]
                assert not np.isfinite(dep).any(), (M, c)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("uplo,tr", [(1, 0), (2, 0), (1, 1)])
def test_ill_conditioned_diagonal_blocks(xk, cplx, uplo, tr):
    """Triangles whose diagonal blocks are far from well conditioned: the
    solve is as backward stable as substitution, componentwise
    |op(T) X - B| <= (M + 8) eps (|op(T)| |X| + |B|), complex four times that."""
    wide = np.clongdouble if cplx else np.longdouble
    for seed, M in enumerate((8, 40, 64, 64, 64, 130)):
        r = np.random.default_rng(100 + seed)
        T = rnd(r, M, M, cplx)
        T[np.arange(M), np.arange(M)] = 0.1j if cplx else 0.1
        Top = OPF[tr](np.tril(T) if uplo == 1 else np.triu(T))
        # a right-hand side whose solution stays of order one
        B = np.asfortranarray((Top.astype(wide) @ rnd(r, M, 21, cplx)).astype(T.dtype))
        X = solve_batch(xk, T, B, uplo, tr, 0)
        res = np.abs(Top.astype(wide) @ X.astype(wide) - B)
        lim = (4 if cplx else 1) * (M + 8) * EPS * (np.abs(Top) @ np.abs(X) + np.abs(B))
        assert (res <= lim).all(), (M, seed, float((res / lim).max()))
