"""Host-side check of the task lists with 64-row panel solves: FINE (FP64: 64 x
64 single-panel updates, 128 x 128 group updates that count for each 64-block)
and HALF (FP32: 128 x 128 updates throughout).  Every task's wait predicate is
met by the tasks before it, and every counter ends at its full value."""
import numpy as np
import pytest

FACT, SOLVE, FINE, HALF = 1, 2, 32, 64
POTRF, TRSM, UPD, FTRSM, FUPD, BTRSM, BUPD, INV = 1, 2, 3, 4, 5, 6, 7, 8


@pytest.mark.parametrize("N,NB,nrhs,G", [(1000, 128, 1, 4), (1153, 128, 70, 4), (700, 64, 3, 8), (1500, 320, 9, 1),
                                         (129, 128, 2, 4), (2000, 256, 0, 2)])
@pytest.mark.parametrize("flag", [FINE, HALF])
@pytest.mark.parametrize("mode", [FACT, FACT | SOLVE, SOLVE])
def test_list_is_deadlock_free(N, NB, nrhs, G, mode, flag):
    import chameleon_b200 as cb
    if mode & SOLVE and nrhs == 0:
        nrhs = 5
    NBB = 64
    NT, NTB = -(-N // NB), -(-nrhs // NBB)
    tm = lambda m: min(NB, N - m * NB)
    b = lambda m: -(-tm(m) // 64)
    cb_ = 64 if flag == FINE else 128            # counted update blocks, substitution rows
    u = lambda m: -(-tm(m) // cb_)
    S = lambda m, n: u(m) * (u(m) + 1) // 2 if m == n else u(m) * u(n)
    ng = lambda n: max(n, 0) if n <= 2 else -(-(n - 2) // G) + 2
    upd, pan = np.zeros((NT, NT), int), np.zeros((NT, NT), int)
    fB, fD, bB, bD = (np.zeros((NT, max(NTB, 1)), int) for _ in range(4))
    fact = bool(mode & FACT)
    for kind, sub, m, n, k, bn, grp in cb.schedule(mode | flag, N, NB, nrhs if mode & SOLVE else 0, NBB, workers=296,
                                                   prof=0 if flag == FINE else 2, kgroup=G):
        if kind == POTRF:
            assert upd[k, k] == ng(k) * S(k, k)
            pan[k, k] += 1
        elif kind == INV:
            pan[k, k] += 1
        elif kind == TRSM:
            assert pan[k, k] == 1 and upd[m, k] == ng(k) * S(m, k) and sub < b(m)
            pan[m, k] += 1
        elif kind == UPD:
            kl, e = k + bn - 1, cb_ if bn == 1 else 128
            assert pan[m, kl] >= b(m) and pan[n, kl] >= b(n) and upd[m, n] >= grp * S(m, n)
            bi, bj = sub & 255, sub >> 8
            r, c = min(e, tm(m) - bi * e), min(e, tm(n) - bj * e)
            assert r > 0 and c > 0
            x, y = -(-r // cb_), -(-c // cb_)
            upd[m, n] += 1 if bn == 1 else (x * (x + 1) // 2 if m == n and bi == bj else x * y)
        elif kind == FTRSM:
            assert pan[k, k] == 1 and fB[k, bn] == k * u(k)
            fD[k, bn] += 1
        elif kind == FUPD:
            assert fD[k, bn] == 1 and (not fact or pan[m, k] == b(m)) and fB[m, bn] >= k * u(m)
            fB[m, bn] += 1
        elif kind == BTRSM:
            assert fD[k, bn] == 1 and bB[k, bn] == (NT - 1 - k) * u(k)
            bD[k, bn] += 1
        elif kind == BUPD:
            assert bD[k, bn] == 1 and bB[m, bn] >= (NT - 1 - k) * u(m)
            bB[m, bn] += 1
    if fact:
        assert all(upd[m, n] == ng(n) * S(m, n) for n in range(NT) for m in range(n, NT))
    if mode & SOLVE:
        assert (bD[:, :NTB] == 1).all()
