"""The pass-pipeline queue of the launch shapes with one sequence a lane (fasttransforms_b200/csrc/
rotations.cu: schedule_passes, shape_pass, shape_split), whose tasks are split into groups of half the
orders, and of the spin transforms' list (the columns of orders -m and m in tasks of their own); restated
with the geometry of tests/test_rot_skew.py:
  * every pass of every group runs once, queued after the group's previous pass;
  * the groups' progress words are disjoint, and fit the words a call on sph, tri and disk plans brings
    (n / 16 + 2 a task, api.cu);
  * the kernel's group g (orders g mod split of task g / split) has the passes it was queued for."""
import pytest

from test_rot_skew import DISK, SPH, SPIN, TRI, default_M, last_order, sequences, step, task_orders, task_sweeps

PASS = {0: 64, 1: 64, 2: 32, 3: 64, 4: 32}      # shape_pass


def task_list(k, M):
    span, mlast = step(k) * task_orders(k), last_order(k, M)
    first = [1] if k == TRI else ([0, 1] if k == SPIN else [2, 3])
    return [mb for f in first for mb in range(f, mlast + 1, span) for _ in range(2 if k == SPIN else 1)]


def schedule(k, M, shape, blk, spin):
    split = sequences(k) if shape in (3, 4) else 1
    orders, tl = task_orders(k) // split, task_list(k, M)
    npass, prog0, nprog = [], [], 0
    for t in range(len(tl) * split):
        mbase = tl[t // split] + step(k) * orders * (t % split)
        nsw = 0 if mbase > last_order(k, M) else task_sweeps(k, M, mbase, blk, spin, orders)[0]
        npass.append(-(-nsw // PASS[shape]))
        prog0.append(nprog)
        nprog += npass[-1]
    q = [(t, prog0[t], r) for r in range(max(npass, default=0)) for t in range(len(npass)) if r < npass[t]]
    return q, npass, nprog, len(tl)


@pytest.mark.parametrize("k,spin", [(SPH, 0), (DISK, 0), (TRI, 0), (SPIN, 0), (SPIN, 2), (SPIN, 5)])
@pytest.mark.parametrize("n", [2, 17, 64, 255, 832, 1024, 4096])
@pytest.mark.parametrize("shape", [0, 2, 3, 4])
@pytest.mark.parametrize("blk", [0, 32])
def test_split_queue(k, spin, n, shape, blk):
    if k == SPIN and blk:
        return
    for M in {default_M(k, n), (default_M(k, n) // 3) | 1}:
        if k == TRI and M != n:
            continue
        q, npass, nprog, ntasks = schedule(k, M, shape, blk, spin)
        at, words = {}, set()
        for i, (t, p0, r) in enumerate(q):
            assert (t, r) not in at and p0 + r not in words
            at[t, r] = i
            words.add(p0 + r)
            assert r == 0 or at[t, r - 1] < i
        assert sorted(at) == sorted((t, r) for t in range(len(npass)) for r in range(npass[t]))
        assert words == set(range(nprog))
        if k != SPIN:
            assert nprog <= ntasks * (n // 16 + 2), (k, n, M, shape)
