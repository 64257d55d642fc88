"""dposv above the order where the substitutions get a launch of their own."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest
import scipy.linalg as sla

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps
UPPER, LOWER = 121, 122
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FRESH = """
import numpy as np, chameleon_b200 as cb
n, nb, nrhs = %d, %d, %d
cb.init()
g = np.random.default_rng(n)
A0 = g.uniform(-0.5, 0.5, (n, n)); A0 = A0 + A0.T + n * np.eye(n)
B0 = g.uniform(-0.5, 0.5, (n, nrhs))
dA, dB = cb.Desc.create(n, n, nb), cb.Desc.create(n, nrhs, nb)
dA.from_numpy(A0); dB.from_numpy(B0)
assert cb.dposv_Tile(cb.ChamLower, dA, dB) == 0
X = dB.to_numpy()
r = np.linalg.norm(B0 - A0 @ X) / (np.linalg.norm(A0) * np.linalg.norm(X))
assert r <= 8 * n * np.finfo(float).eps, r
"""


def run_fresh(code):
    subprocess.run([sys.executable, "-c", code], cwd=ROOT, check=True, timeout=300)


@pytest.mark.parametrize("n,nb,nrhs", [(3144, 262, 64), (3200, 200, 900)])
def test_first_call_of_a_process(n, nb, nrhs):
    """The substitutions need more counters than the factorization, and no
    earlier call has grown the workspace."""
    run_fresh(FRESH % (n, nb, nrhs))


SCARCE = """
import numpy as np, chameleon_b200 as cb
n, nb, nrhs, mib, potrs, want = %r
cb.init()
g = np.random.default_rng(n)
A0 = g.uniform(-0.5, 0.5, (n, n)); A0 = A0 + A0.T + n * np.eye(n)
B0 = g.uniform(-0.5, 0.5, (n, nrhs))
dA, dB = cb.Desc.create(n, n, nb), cb.Desc.create(n, nrhs, nb)
dA.from_numpy(A0); dB.from_numpy(B0)
if potrs:
    assert cb.dpotrf_Tile(cb.ChamLower, dA) == 0
L = cb.lib()
L.CHAM_B200_Workspace_Limit(int(mib * 2**20))
rc = (cb.dpotrs_Tile if potrs else cb.dposv_Tile)(cb.ChamLower, dA, dB)
assert rc == want, rc
L.CHAM_B200_Workspace_Limit(-1)
if want:   # nothing was started
    assert np.array_equal(dB.to_numpy(), B0) and (potrs or np.array_equal(dA.to_numpy(), A0))
    assert (cb.dpotrs_Tile if potrs else cb.dposv_Tile)(cb.ChamLower, dA, dB) == 0
X = dB.to_numpy()
r = np.linalg.norm(B0 - A0 @ X) / (np.linalg.norm(A0) * np.linalg.norm(X))
assert r <= 8 * n * np.finfo(float).eps, r
"""


@pytest.mark.parametrize("potrs", [False, True])
@pytest.mark.parametrize("mib,want", [(8, 0), (0.01, -106)])
def test_little_memory(mib, want, potrs):
    """Tile inverses and forward results take 35 MiB here: without them the call
    runs as one launch, and without room for that it leaves A and B alone."""
    run_fresh(SCARCE % ((3200, 200, 1000, mib, potrs, want),))


SCARCE_INVERSE = """
import numpy as np, torch, chameleon_b200 as cb
n = 1500
cb.init()
T = np.tril(np.random.default_rng(n).uniform(-0.5, 0.5, (n, n)) / n) + np.eye(n)
for uplo, F in ((cb.ChamLower, T), (cb.ChamUpper, T.T)):
    R = np.linalg.inv(F)
    W = np.asfortranarray(F.copy())
    cb.dlauum(uplo, 8, np.eye(8, order="F"), 8)      # the context's first allocations
    V = np.asfortranarray(F.copy())
    S = np.asfortranarray(F.copy()); S[700, 700] = 0.0
    dev = [torch.from_numpy(a.T.copy()).cuda() for a in (W, V, S)]
    cb.lib().CHAM_B200_Workspace_Limit(24 << 20)     # one N x N workspace (18 MiB), not two
    assert cb.dtrtri(uplo, cb.ChamNonUnit, n, dev[0], n) == 0
    assert cb.dpotri(uplo, n, dev[1], n) == 0
    assert cb.dtrtri(uplo, cb.ChamNonUnit, n, dev[2], n) == 701
    cb.lib().CHAM_B200_Workspace_Limit(-1)
    W, V, Z = (d.cpu().numpy().T for d in dev)
    tri = np.tril if uplo == cb.ChamLower else np.triu
    bound = 8 * n * np.finfo(float).eps
    assert np.abs(W - F + tri(F) - tri(R)).max() <= bound
    P = R.T @ R if uplo == cb.ChamLower else R @ R.T
    assert np.abs(tri(V) - tri(P)).max() <= bound * 4
    assert np.array_equal(Z, S)
"""


def test_inverses_with_one_workspace():
    run_fresh(SCARCE_INVERSE)


def kernel_matrix(n, length, nugget, seed):
    """Covariance of a Gaussian kernel on sorted points: ill-conditioned diagonal tiles."""
    x = np.sort(np.random.default_rng(seed).uniform(0, 1, n))
    return np.exp(-0.5 * ((x[:, None] - x) / length) ** 2) + nugget * np.eye(n)


def block_inverse(L, w=8):
    """L^-1 by block rows of w, as the 64 x 64 leaf makes it."""
    X = np.zeros_like(L)
    for p in range(0, len(L), w):
        q = slice(p, min(p + w, len(L)))
        X[q, q] = sla.solve_triangular(L[q, q], np.eye(q.stop - p), lower=True)
        X[q, :p] = -X[q, q] @ (L[q, :p] @ X[:p, :p])
    return X


def solve_by_blocks(L, B, h=64):
    """L L^T X = B with explicit inverses of the h x h diagonal blocks alone."""
    Y, n = B.copy(), len(L)
    inv = [block_inverse(L[j:j + h, j:j + h]) for j in range(0, n, h)]
    for j in range(0, n, h):
        Y[j:j + h] = inv[j // h] @ (Y[j:j + h] - L[j:j + h, :j] @ Y[:j])
    for j in reversed(range(0, n, h)):
        Y[j:j + h] = inv[j // h].T @ (Y[j:j + h] - L[j + h:, j:j + h].T @ Y[j + h:])
    return Y


def backward_error(A, X, B):
    return np.abs(B - A @ X).max() / (np.abs(A).sum(1).max() * np.abs(X).max())


@pytest.mark.parametrize("n,nb,nrhs,uplo", [(512, 512, 3, LOWER), (700, 350, 40, UPPER), (1000, 384, 9, LOWER),
                                            (3073, 512, 5, UPPER), (2048, 200, 70, LOWER)])
@pytest.mark.parametrize("length,nugget", [(0.02, 1e-10), (0.1, 1e-8), (0.02, 1e-4)])
def test_backward_error_of_ill_conditioned_potrs(cb, n, nb, nrhs, uplo, length, nugget):
    """No further from backward stability than inverted 64 x 64 blocks are
    (within 4 x: another order of the same sums), whatever the condition."""
    A = kernel_matrix(n, length, nugget, n)
    L = np.linalg.cholesky(A)
    A = L @ L.T
    B = A @ np.random.default_rng(nb).standard_normal((n, nrhs))
    F = np.where(np.tri(n, dtype=bool), L, np.nan)
    F = F if uplo == LOWER else F.T
    dA, dB = cb.Desc.create(n, n, nb), cb.Desc.create(n, nrhs, nb)
    dA.from_numpy(F)
    dB.from_numpy(B)
    assert cb.dpotrs_Tile(uplo, dA, dB) == 0
    got, ref = backward_error(A, dB.to_numpy(), B), backward_error(A, solve_by_blocks(L, B), B)
    assert got <= 4 * ref + 4 * EPS, (got, ref)


@pytest.mark.parametrize("n", [2000, 3100, 4096])
def test_backward_error_of_ill_conditioned_posv(cb, n):
    A = kernel_matrix(n, 0.02, 1e-8, n)
    B = A @ np.random.default_rng(n).standard_normal((n, 4))
    dA, dB = cb.Desc.create(n, n, 512), cb.Desc.create(n, 4, 512)
    dA.from_numpy(A)
    dB.from_numpy(B)
    assert cb.dposv_Tile(LOWER, dA, dB) == 0
    got = backward_error(A, dB.to_numpy(), B)
    ref = backward_error(A, solve_by_blocks(np.linalg.cholesky(A), B), B)
    assert got <= 4 * ref + 4 * EPS, (got, ref)


@pytest.mark.parametrize("uplo", [LOWER, UPPER])
def test_nan_in_a_factor_reaches_the_solution_it_belongs_to(cb, uplo):
    """A NaN in the last diagonal tile of the factor spoils that tile's rows and,
    through the backward sweep, those above: no stale or partial result."""
    n, nb = 1024, 256
    L = np.linalg.cholesky(kernel_matrix(n, 0.02, 1e-2, 5))
    L[n - 1, n - 1] = np.nan
    dA, dB = cb.Desc.create(n, n, nb), cb.Desc.create(n, 2, nb)
    dA.from_numpy(L if uplo == LOWER else L.T.copy())
    dB.from_numpy(np.ones((n, 2)))
    assert cb.dpotrs_Tile(uplo, dA, dB) == 0
    assert np.isnan(dB.to_numpy()[n - 1]).all()


@pytest.mark.parametrize("n,nb,nrhs,array,uplo", [(2048, 512, 40001, True, LOWER), (1000, 200, 50003, False, UPPER),
                                                  (700, 250, 75001, False, LOWER)])
@pytest.mark.parametrize("posv", [False, True])
def test_wide_right_hand_sides(cb, n, nb, nrhs, array, uplo, posv):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    S = torch.rand((n, n), dtype=torch.float64, device="cuda", generator=g).sub_(0.5)
    S = S + S.T + n * torch.eye(n, dtype=torch.float64, device="cuda")
    F = torch.linalg.cholesky(S)                     # lower; torch rows are our columns
    a = (S if posv else F.T if uplo == LOWER else F).clone(memory_format=torch.contiguous_format)
    b0 = torch.rand((nrhs, n), dtype=torch.float64, device="cuda", generator=g).sub_(0.5)
    b, ptr = b0.clone(), lambda t: ctypes.c_void_p(t.data_ptr())
    if array:
        assert (cb.dposv if posv else cb.dpotrs)(uplo, n, nrhs, a, n, b, n) == 0
    else:
        L, dA, dB = cb.lib(), cb.Desc.create(n, n, nb), cb.Desc.create(n, nrhs, nb)
        assert L.CHAMELEON_Lap2Desc(123, ptr(a), n, dA.ptr) == 0 and L.CHAMELEON_Lap2Desc(123, ptr(b), n, dB.ptr) == 0
        assert (cb.dposv_Tile if posv else cb.dpotrs_Tile)(uplo, dA, dB) == 0
        assert L.CHAMELEON_Desc2Lap(123, dB.ptr, ptr(b), n) == 0
    r = float(torch.linalg.norm(b @ S - b0) / (torch.linalg.norm(S) * torch.linalg.norm(b)))
    assert r <= 8 * n * EPS


@pytest.mark.parametrize("bad", [1, 40, 3050])
@pytest.mark.parametrize("uplo", [LOWER, UPPER])
def test_failed_factorization_leaves_the_right_hand_sides(cb, uplo, bad):
    """The substitutions' launch sees that the factorization's has failed."""
    n, nb = 3100, 512
    A = np.random.default_rng(1).uniform(-0.5, 0.5, (n, n)) + n * np.eye(n)
    A[bad - 1, bad - 1] = -1.0
    B = np.random.default_rng(2).uniform(-0.5, 0.5, (n, 7))
    dA, dB = cb.Desc.create(n, n, nb), cb.Desc.create(n, 7, nb)
    dA.from_numpy(A)
    dB.from_numpy(B)
    assert cb.dposv_Tile(uplo, dA, dB) == bad
    assert np.array_equal(dB.to_numpy(), B)
    dA.from_numpy(n * np.eye(n))               # and the next call is not affected
    assert cb.dposv_Tile(uplo, dA, dB) == 0
    assert np.abs(dB.to_numpy() * n - B).max() <= 4 * EPS


@pytest.mark.parametrize("n,nb,nrhs", [(3073, 512, 1), (3200, 200, 17), (3144, 262, 64), (3100, 509, 33)])
@pytest.mark.parametrize("uplo", [LOWER, UPPER])
@pytest.mark.parametrize("layout", ["tiles", "array"])
def test_two_launches_over_tilings(cb, layout, uplo, n, nb, nrhs):
    """Remainders, tiles with and without usable divisors, odd leading dimension."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    ld = n + 3
    S = torch.rand((n, n), dtype=torch.float64, device="cuda", generator=g).sub_(0.5)
    S = S + S.T + n * torch.eye(n, dtype=torch.float64, device="cuda")
    B = torch.rand((nrhs, n), dtype=torch.float64, device="cuda", generator=g).sub_(0.5)
    part = S.triu() if uplo == LOWER else S.tril()     # rows are columns
    a = torch.full((n, ld), float("nan"), dtype=torch.float64, device="cuda")
    a[:, :n] = torch.where(part != 0, part, a[:, :n])
    b = torch.full((nrhs, ld), float("nan"), dtype=torch.float64, device="cuda")
    b[:, :n] = B
    p, L = lambda t: ctypes.c_void_p(t.data_ptr()), cb.lib()
    if layout == "tiles":
        dA, dB = cb.Desc.create(n, n, nb), cb.Desc.create(n, nrhs, nb)
    for step in ("posv", "potrs"):
        b[:, :n] = B
        if layout == "array":
            assert (cb.dposv if step == "posv" else cb.dpotrs)(uplo, n, nrhs, a, ld, b, ld) == 0
        else:
            if step == "posv":
                assert L.CHAMELEON_Lap2Desc(123, p(a), ld, dA.ptr) == 0
            assert L.CHAMELEON_Lap2Desc(123, p(b), ld, dB.ptr) == 0
            assert (cb.dposv_Tile if step == "posv" else cb.dpotrs_Tile)(uplo, dA, dB) == 0
            assert L.CHAMELEON_Desc2Lap(123, dB.ptr, p(b), ld) == 0
        X = b[:, :n]
        r = float(torch.linalg.norm(X @ S - B) / (torch.linalg.norm(S) * torch.linalg.norm(X)))
        assert r <= 8 * n * EPS, (step, r)


def test_trace_holds_both_launches(cb):
    """The substitutions' records follow the factorization's."""
    rec = np.dtype([("task", "<i4"), ("smid", "<i4"), ("t0", "<u8"), ("t1", "<u8"), ("wait", "<u4"), ("ph", "<u4", 3)])
    n, cap, L = 3100, 40000, cb.lib()
    dA, dB = cb.Desc.create(n, n, 512), cb.Desc.create(n, 5, 512)
    dA.from_numpy(n * np.eye(n))
    dB.from_numpy(np.ones((n, 5)))
    assert L.CHAM_B200_Trace_Enable(cap) == 0
    try:
        assert cb.dposv_Tile(LOWER, dA, dB) == 0
        out = np.zeros(cap, rec)
        assert L.CHAM_B200_Trace_Read(out.ctypes.data_as(ctypes.c_void_p), cap) == 0
    finally:
        L.CHAM_B200_Trace_Enable(0)
    used = int((out["t1"] > 0).sum())
    starts = np.flatnonzero(out["task"][:used] == 0)
    assert (out["t1"][:used] > 0).all() and len(starts) == 2, used
    k = int(starts[1])
    assert np.array_equal(out["task"][:k], np.arange(k)) and np.array_equal(out["task"][k:used], np.arange(used - k))
    assert out["t1"][:k].max() <= out["t0"][k:used].min()
