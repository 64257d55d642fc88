"""FP64 executor tiles finer than the storage's, and the 64 x 64 leaf.

The executor picks its own tile size inside the storage tiles (any size for
column-major storage, a divisor of the tile otherwise): every layout, triangle
and remainder is checked against numpy's factor and solution.  Errors are
bounded by the backward error of Cholesky and of the two substitutions,
a small multiple of n eps relative to the norms (Higham, Accuracy and
Stability of Numerical Algorithms, theorems 10.3 and 10.4): 8 n eps.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps
UPPER, LOWER = 121, 122


def spd(n, seed, scale=1.0):
    g = np.random.default_rng(seed)
    a = g.uniform(-0.5, 0.5, (n, n))
    return (a + a.T + n * np.eye(n)) * scale


@pytest.mark.parametrize("layout", ["tiles", "array"])
@pytest.mark.parametrize("uplo", [UPPER, LOWER])
@pytest.mark.parametrize("n,nb,nrhs", [(1, 64, 1), (127, 512, 2), (129, 512, 9), (385, 128, 1), (700, 320, 70),
                                       (641, 200, 8), (300, 7, 3), (1031, 384, 65), (1152, 512, 33)])
def test_posv_and_potrs_over_tilings(cb, layout, uplo, n, nb, nrhs):
    import torch
    A0 = spd(n, n + nb)
    B0 = np.random.default_rng(nb).uniform(-0.5, 0.5, (n, nrhs))
    poisoned = np.where(np.tri(n, k=0 if uplo == LOWER else -1, dtype=bool) == (uplo == LOWER), A0, np.nan)
    if layout == "array":   # torch (columns, rows): column-major storage
        tA, tB = torch.from_numpy(poisoned.T.copy()).cuda(), torch.from_numpy(B0.T.copy()).cuda()
        dA, dB = cb.Desc.create(n, n, nb, mat=tA), cb.Desc.create(n, nrhs, nb, mat=tB)
    else:
        dA, dB = cb.Desc.create(n, n, nb), cb.Desc.create(n, nrhs, nb)
        dA.from_numpy(poisoned)
        dB.from_numpy(B0)
    get = (lambda: (tA.cpu().numpy().T, tB.cpu().numpy().T)) if layout == "array" else (
        lambda: (dA.to_numpy(uplo), dB.to_numpy()))
    X = np.linalg.solve(A0, B0)
    for step in ("posv", "potrs"):
        if step == "potrs":
            if layout == "array":
                tB.copy_(torch.from_numpy(B0.T.copy()))
            else:
                dB.from_numpy(B0)
        assert (cb.dposv_Tile if step == "posv" else cb.dpotrs_Tile)(uplo, dA, dB) == 0
        F, Y = get()
        L = np.tril(F) if uplo == LOWER else np.triu(F).T
        assert np.linalg.norm(A0 - L @ L.T) <= 8 * n * EPS * np.linalg.norm(A0)
        assert np.linalg.norm(Y - X) <= 8 * n * EPS * np.linalg.cond(A0) * np.linalg.norm(X)
        if layout == "array" and n > 1:   # the other triangle is not written
            off = np.triu(F, 1) if uplo == LOWER else np.tril(F, -1)
            assert np.isnan(off[off != 0]).all()


@pytest.mark.parametrize("n,scale", [(n, 1.0) for n in (1, 7, 8, 9, 31, 33, 56, 57, 64, 65, 72, 128)] +
                         [(40, 1e-290), (64, 1e290), (23, 3e-309)])
@pytest.mark.parametrize("uplo", [UPPER, LOWER])
def test_tile_potrf_fp64_orders_and_scales(cb, uplo, n, scale):
    """Every remainder of the 8-wide panels, and pivots beyond the range of
    the reciprocal estimates (3e-309: the entries off the diagonal are subnormal,
    absolute errors of a few subnormal units, relative to the scale, bound it)."""
    import torch
    L = cb.lib()
    A0 = spd(n, 3 * n, scale)
    t = torch.from_numpy(A0.T.copy()).cuda()
    info = torch.full((1,), -7, dtype=torch.int32, device="cuda")
    h = ctypes.c_void_p()
    assert L.CHAM_B200_Handle_Create(ctypes.byref(h), None) == 0
    assert L.CUDA_dpotrf(uplo, n, t.data_ptr(), n, None, 0, info.data_ptr(), h) == 0
    torch.cuda.synchronize()
    L.CHAM_B200_Handle_Destroy(h)
    assert int(info) == 0
    F = t.cpu().numpy().T
    Lf = np.tril(F) if uplo == LOWER else np.triu(F).T
    # in units of the scale, so that the squares stay representable
    r = np.sqrt(scale)
    err = np.abs(A0 / scale - (Lf / r) @ (Lf / r).T).max() / n
    assert err <= 8 * n * EPS + 8 * 4.94e-324 / scale


@pytest.mark.parametrize("n", [1, 9, 64, 100, 256])
@pytest.mark.parametrize("scale", [1.0, 1e-34, 1e34])
def test_tile_potrf_fp32_scales(cb, n, scale):
    import torch
    L = cb.lib()
    A0 = spd(n, 5 * n, scale).astype(np.float32)
    t = torch.from_numpy(A0.T.copy()).cuda()
    info = torch.full((1,), -7, dtype=torch.int32, device="cuda")
    h = ctypes.c_void_p()
    assert L.CHAM_B200_Handle_Create(ctypes.byref(h), None) == 0
    assert L.CUDA_spotrf(LOWER, n, t.data_ptr(), n, None, 0, info.data_ptr(), h) == 0
    torch.cuda.synchronize()
    L.CHAM_B200_Handle_Destroy(h)
    assert int(info) == 0
    Lf = np.tril(t.cpu().numpy().T).astype(np.float64)
    err = np.abs(A0.astype(np.float64) - Lf @ Lf.T).max() / (n * scale)
    # FP32 FMA throughout at these orders: n-term sums
    assert err <= 8 * n * 2.0 ** -24


@pytest.mark.parametrize("n,bad", [(64, 1), (64, 9), (64, 64), (130, 65), (200, 129), (200, 200)])
def test_first_non_positive_pivot(cb, n, bad):
    import torch
    A0 = spd(n, n)
    A0[bad - 1, bad - 1] = -1.0
    t = torch.from_numpy(A0.copy()).cuda()
    assert cb.dpotrf(LOWER, n, t, n) == bad


def factor(cb, name, a):
    """The lower factor of one tile call and its info."""
    import torch
    L = cb.lib()
    t = torch.from_numpy(a.T.copy()).cuda()
    info = torch.full((1,), -7, dtype=torch.int32, device="cuda")
    h = ctypes.c_void_p()
    assert L.CHAM_B200_Handle_Create(ctypes.byref(h), None) == 0
    n = a.shape[0]
    assert getattr(L, name)(LOWER, n, t.data_ptr(), n, None, 0, info.data_ptr(), h) == 0
    torch.cuda.synchronize()
    L.CHAM_B200_Handle_Destroy(h)
    return np.tril(t.cpu().numpy().T), int(info)


@pytest.mark.parametrize("n", [1, 5, 64])
@pytest.mark.parametrize("name,dtype,d", [("CUDA_dpotrf", np.float64, 1e-310), ("CUDA_dpotrf", np.float64, 5e-324),
                                          ("CUDA_spotrf", np.float32, 1e-39), ("CUDA_spotrf", np.float32, 1e-45)])
def test_subnormal_pivots(cb, n, name, dtype, d):
    """Diagonal matrices whose pivots' reciprocals overflow: the roots are exact
    to one rounding, and nothing spreads to the zeros or to the padding."""
    a = np.diag(np.full(n, d, dtype))
    F, info = factor(cb, name, a)
    assert info == 0
    assert np.abs(np.diag(F) / np.sqrt(np.diag(a)) - 1).max() <= 2 * np.finfo(dtype).eps
    assert (F[~np.eye(n, dtype=bool)] == 0).all()


@pytest.mark.parametrize("name,dtype", [("CUDA_dpotrf", np.float64), ("CUDA_spotrf", np.float32)])
@pytest.mark.parametrize("n,at", [(1, 0), (24, 3), (64, 63), (64, 40)])
def test_infinite_pivot(cb, n, at, name, dtype):
    """An infinite diagonal entry of a diagonal matrix, as LAPACK factors it."""
    a = np.diag(np.full(n, 4.0, dtype))
    a[at, at] = np.inf
    F, info = factor(cb, name, a)
    assert info == 0
    want = np.diag(np.full(n, 2.0, dtype))
    want[at, at] = np.inf
    assert np.array_equal(F, want)


def test_fp32_leaf_rounds_an_entry_about_once(cb):
    """Dominant diagonal: what is subtracted from an entry is small, so that its
    error is that of the last rounding, 2^-24 at most (sums of 64 single
    subtractions at the entry's size gave 1.4 times that)."""
    errs = []
    for seed in range(8):
        a = spd(64, seed).astype(np.float32)
        F, info = factor(cb, "CUDA_spotrf", a)
        assert info == 0
        R = np.linalg.cholesky(a.astype(np.float64))
        errs.append(np.linalg.norm(F - R) / np.linalg.norm(R))
    assert np.mean(errs) <= 2.0 ** -24


@pytest.mark.parametrize("fp32", [False, True])
def test_pivot_estimates(cb, fp32):
    """1 / d and d^(-1/2) over the accepted exponents: one rounding and what the
    series leaves out, and for the root half a rounding of d q (rec.cuh)."""
    import torch
    dt, u, lo, hi = (np.float32, 2.0 ** -24, 1e-30, 1e30) if fp32 else (np.float64, 2.0 ** -53, 1e-280, 1e280)
    g = np.random.default_rng(3)
    n = 1 << 18
    d = np.concatenate([np.exp(g.uniform(np.log(lo), np.log(hi), n)), g.uniform(1, 4, n), 1 + g.uniform(0, 1e-6, n),
                        4 - g.uniform(0, 1e-6, n), 2.0 ** g.integers(-90, 90, n)]).astype(dt)
    bad = np.array([0.0, -1.0, np.nan, np.inf, -np.inf, lo / 2, hi * 2], dt)
    x = torch.from_numpy(np.concatenate([d, bad])).cuda()
    rc, rs, ok = torch.empty_like(x), torch.empty_like(x), torch.empty(x.numel(), dtype=torch.int32, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    torch.cuda.synchronize()
    assert cb.lib().CHAM_B200_Test_Pivot_Recip(int(fp32), x.numel(), p(x), p(rc), p(rs), p(ok)) == 0
    used = ok.cpu().numpy().astype(bool)
    assert used[:len(d)][(d > lo) & (d < hi)].all() and not used[len(d):].any()
    t = d.astype(np.longdouble)
    use = used[:len(d)]
    erc = np.abs(rc.cpu().numpy()[:len(d)].astype(np.longdouble) * t - 1)[use].max()
    ers = np.abs(rs.cpu().numpy()[:len(d)].astype(np.longdouble) * np.sqrt(t) - 1)[use].max()
    assert erc <= 1.01 * u and ers <= 1.6 * u, (erc / u, ers / u)


@pytest.mark.parametrize("n", [512, 300, 129, 100])
def test_potrf_under_stream_capture(cb, n):
    """A handle that has factored order 512 is captured at that order and at
    smaller ones it has not seen; the graph factors what its replays find."""
    import torch
    L, h, s = cb.lib(), ctypes.c_void_p(), torch.cuda.Stream()
    assert L.CHAM_B200_Handle_Create(ctypes.byref(h), ctypes.c_void_p(s.cuda_stream)) == 0
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    info = torch.full((1,), -7, dtype=torch.int32, device="cuda")
    warm = torch.from_numpy(spd(512, 1).T.copy()).cuda()
    torch.cuda.synchronize()
    assert L.CUDA_dpotrf(LOWER, 512, p(warm), 512, None, 0, p(info), h) == 0
    t = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        assert L.CUDA_dpotrf(LOWER, n, p(t), n, None, 0, p(info), h) == 0
    for seed in (5, 6):
        A0 = spd(n, seed)
        t.copy_(torch.from_numpy(A0.T.copy()))
        info.fill_(-7)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        F = np.tril(t.cpu().numpy().T)
        assert int(info) == 0
        assert np.linalg.norm(A0 - F @ F.T) <= 8 * n * EPS * np.linalg.norm(A0)
    del graph
    torch.cuda.synchronize()
    L.CHAM_B200_Handle_Destroy(h)


@pytest.mark.parametrize("n,w", [(1, 1), (64, 3), (65, 9), (513, 130), (200, 2369), (3072, 5), (3073, 2), (1000, 2500)])
@pytest.mark.parametrize("side", [141, 142])
@pytest.mark.parametrize("uplo,trans,diag,alpha", [(LOWER, 111, 131, 1.0), (LOWER, 112, 132, -0.5), (UPPER, 111, 132, 2.0),
                                                   (UPPER, 112, 131, 0.0)])
def test_trsm_routes(cb, n, w, side, uplo, trans, diag, alpha):
    """Strips, and the 64-column route beyond their order and width."""
    import torch
    g = np.random.default_rng(n + w)
    T = g.uniform(-0.5, 0.5, (n, n)) / n
    T[np.diag_indices(n)] = g.uniform(1, 2, n)
    tri = np.tril if uplo == LOWER else np.triu
    full = tri(T).copy()
    if diag == 132:
        full[np.diag_indices(n)] = 1.0
        T[np.diag_indices(n)] = np.nan                     # not referenced
    A = np.where(tri(np.ones((n, n), bool)), T, np.nan)
    rows, cols = (n, w) if side == 141 else (w, n)
    B = g.uniform(-0.5, 0.5, (rows, cols))
    op = full if trans == 111 else full.T
    want = alpha * (np.linalg.solve(op, B) if side == 141 else np.linalg.solve(op.T, B.T).T)
    a, b = torch.from_numpy(A.T.copy()).cuda(), torch.from_numpy(B.T.copy()).cuda()
    L, h = cb.lib(), ctypes.c_void_p()
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    assert L.CHAM_B200_Handle_Create(ctypes.byref(h), None) == 0
    torch.cuda.synchronize()
    assert L.CUDA_dtrsm(side, uplo, trans, diag, rows, cols, ctypes.byref(ctypes.c_double(alpha)), p(a), n, p(b), rows,
                        h) == 0
    torch.cuda.synchronize()
    L.CHAM_B200_Handle_Destroy(h)
    # row sums of |T^-1| |T| are below 4: a few eps each, whatever n
    assert np.abs(b.cpu().numpy().T - want).max() <= 64 * EPS * np.abs(want).max()
