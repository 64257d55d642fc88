"""Host-side checks of what one executor call plans before it launches anything."""
import ctypes

import numpy as np
import pytest

FACT, SOLVE = 1, 2
# columns of a planned launch (0, 1: tile size, column block)
CTR, INV, XINV, Y, MODE, GROUP = 2, 3, 4, 5, 6, 7


def plan(mode, N, nb, nrhs, array=False, nbb=None, fp32=False):
    import chameleon_b200 as cb
    launch, res = np.zeros((2, 8), np.int64), np.zeros(4, np.int64)
    p = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_int64))
    n = cb.lib().CHAM_B200_Exec_Plan(mode, N, nb, int(array), nrhs, nbb or nb, int(fp32), p(launch), p(res))
    return launch[:n], res


@pytest.mark.parametrize("N,nb,nrhs", [(3144, 262, 64), (3200, 200, 900), (3073, 512, 1), (8192, 512, 64),
                                       (5003, 384, 17), (2048, 320, 1)])
@pytest.mark.parametrize("array", [False, True])
def test_workspace_is_reserved_for_every_launch(N, nb, nrhs, array):
    """The factorization's launch still runs when the substitutions' is
    enqueued, so no buffer may grow between the two: what the call reserves
    before the first launch covers both."""
    launch, res = plan(FACT | SOLVE, N, nb, nrhs, array)
    assert len(launch) == (2 if N > 3072 else 1)
    assert (res >= launch[:, CTR:MODE].max(axis=0)).all()


def test_substitutions_may_need_more_counters_than_the_factorization():
    launch, res = plan(FACT | SOLVE, 3144, 262, 64)
    assert launch[1, CTR] > launch[0, CTR]
    assert res[0] == launch[1, CTR] and res[1] == launch[0, INV]


@pytest.mark.parametrize("bad", [-1, 0, 1, 3])
def test_a_failed_launch_is_not_left_behind(bad):
    """After a step that fails nothing more is enqueued, and what was is waited for."""
    import chameleon_b200 as cb
    calls, n = (ctypes.c_int * 8)(), ctypes.c_int()
    rc = cb.lib().CHAM_B200_Test_Enqueue_All(4, bad, 103, calls, ctypes.byref(n))
    last = 3 if bad < 0 else bad
    assert rc == (0 if bad < 0 else 103)
    assert list(calls[:n.value]) == [*range(last + 1), -1]


@pytest.mark.parametrize("n", [1, 128, 129, 512, 4096])
@pytest.mark.parametrize("device", [0, 1, 3])
def test_dpotrf_of_another_device_keeps_to_its_own_memory(n, device):
    """Task lists and executor workspaces are on the library's device: a stream
    of another one runs the kernel that uses the handle's memory alone."""
    import chameleon_b200 as cb
    on = cb.lib().CHAM_B200_Test_Potrf_On_Dag
    assert on(n, device, device) == (n > 128)
    assert not any(on(n, device, d) for d in (-1, 0, 1, 2, 3) if d != device)


@pytest.mark.parametrize("nb", [16383, 16411, 30011])
def test_blocks_of_a_large_tile_fit_the_task(nb):
    """Storage tiles without a usable divisor are executor tiles: their blocks'
    indices (8 bits each) must tell all of them apart."""
    import chameleon_b200 as cb
    N = 2 * nb
    launch, _ = plan(FACT, N, nb, 0)
    NB, mode = int(launch[0, 0]), int(launch[0, MODE])
    t = cb.schedule(mode, N, NB, 0, NB, workers=296, kgroup=1)
    e = 64 if mode & 32 else 128
    upd = t[t[:, 0] == 3]
    subs = {(m, n, k): [] for m, n, k in upd[:, 2:5].tolist()}
    for _, sub, m, n, k, _, _ in upd.tolist():
        subs[m, n, k].append(sub & 0xffff)
    rows = lambda m: min(NB, N - m * NB)
    blk = lambda m: -(-rows(m) // e)
    for (m, n, k), got in subs.items():
        want = blk(m) * (blk(m) + 1) // 2 if m == n else blk(m) * blk(n)
        assert len(set(got)) == len(got) == want
        assert max(x & 255 for x in got) == blk(m) - 1
    pan = t[t[:, 0] == 2]
    assert (pan[:, 1] >= 0).all() and (pan[:, 1] * e < NB).all()


@pytest.mark.parametrize("n,nb,array,few,many", [(4096, 384, True, 12000, 30000), (8192, 512, False, 8192, 16384),
                                                 (8192, 250, False, 3000, 7000), (2048, 384, True, 300, 45000)])
def test_wide_right_hand_sides_take_no_second_array(n, nb, array, few, many):
    """Past the width where 128-row tasks are faster the substitutions run on the
    storage's tiles, without tile inverses and without an array of B's size."""
    FINE, XINV_MODE = 32, 4
    for mode in (SOLVE, FACT | SOLVE):
        a, _ = plan(mode, n, nb, few, array)
        b, _ = plan(mode, n, nb, many, array)
        assert a[-1, MODE] & FINE and (mode == SOLVE) <= (a[-1, Y] == 8 * n * few)
        assert not b[-1, MODE] & (FINE | XINV_MODE) and b[-1, Y] == b[-1, XINV] == 0
        assert b[-1, 0] == (384 if array else nb)
        assert len(b) == (1 if mode == SOLVE else 2)


@pytest.mark.parametrize("nb,line", [(128, 20480), (256, 20480), (384, 30720), (512, 30720)])
def test_update_groups_of_the_tensor_core_path(nb, line):
    HALF = 64
    for n, half, group in ((line, True, 8), (line + nb, False, 12)):
        a, _ = plan(FACT, n, nb, 0, fp32=True)
        assert bool(a[0, MODE] & HALF) == half and a[0, GROUP] == group


def test_task_list_of_a_large_order_fits_a_small_process():
    """The host's task graph has a task per update group, not per update: order
    65536 in 1 GB of address space beyond the process's own."""
    import os
    import subprocess
    import sys
    code = """
import resource, chameleon_b200 as cb
L = cb.lib()
have = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (have + (1 << 30),) * 2)
assert L.CHAM_B200_Schedule_Size(1 | 32, 65536, 128, 0, 128, 296, 0, 32) > 0
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", code], cwd=root, check=True, timeout=300)


@pytest.mark.parametrize("n,nrhs,launches", [(100, 400001, 1), (256, 150000, 1), (500, 70000, 2), (2048, 16385, 2),
                                             (2048, 64, 1), (3073, 1, 2)])
def test_launches_of_a_solve(n, nrhs, launches):
    """Two where B outweighs the factorization of more than two tiles, or above 3072."""
    assert len(plan(FACT | SOLVE, n, 384, nrhs, array=True)[0]) == launches
