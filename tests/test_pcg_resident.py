"""The standalone solve on one block an SM (pcg_resident): sizes around its
blocks and rows a thread, rows of uneven length up to ones that do not fit the
shared memory, empty systems' corner values, and calls from several threads."""
import threading

import numpy as np
import pytest

import tetfit_b200 as tb

pytestmark = pytest.mark.gpu


def spd(n, seed, long_rows=0, band=3):
    """Random symmetric, diagonally dominant CSR: `band` couplings a row, and
    `long_rows` rows that couple to 300 others."""
    r = np.random.default_rng(seed)
    i = np.repeat(np.arange(n), band)
    j = np.minimum(n - 1, i + r.integers(1, max(2, n // 7), len(i)))
    if long_rows:
        big = r.choice(n, long_rows, replace=False)
        i = np.concatenate([i, np.repeat(big, 300)])
        j = np.concatenate([j, r.integers(0, n, 300 * long_rows)])
    i, j = i[i != j], j[i != j]
    key = np.unique(np.minimum(i, j) * n + np.maximum(i, j))
    i, j = key // n, key % n
    v = -r.uniform(0.1, 1.0, len(key))
    diag = np.full(n, 0.2) + r.uniform(0, 0.3, n)
    np.add.at(diag, i, -v)
    np.add.at(diag, j, -v)
    rows = np.concatenate([i, j, np.arange(n)])
    cols = np.concatenate([j, i, np.arange(n)])
    vals = np.concatenate([v, v, diag])
    o = np.lexsort((cols, rows))
    ptr = np.zeros(n + 1, dtype=np.int64)
    ptr[1:] = np.cumsum(np.bincount(rows, minlength=n))
    return ptr, cols[o].astype(np.int32), vals[o]


def check(ptr, col, val, seed, tol=1e-10, guess=False):
    import torch
    n = len(ptr) - 1
    dev = torch.device("cuda:0")
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    r = np.random.default_rng(seed)
    b = r.standard_normal(n)
    x = t(r.standard_normal(n) if guess else np.zeros(n))
    rc, it, rs = tb.pcg_solve(t(ptr), t(col), t(val), t(b), x, tol=tol, maxiter=1000, criterion=1)
    assert rc == tb.TF_OK, tb.last_thread_error()
    xs = x.cpu().numpy()
    res = b.copy()
    np.add.at(res, np.repeat(np.arange(n), np.diff(ptr)), -val * xs[col])
    # the recurrence's residual stops at tol; the true one drifts by rounding only
    assert np.linalg.norm(res) <= 2 * tol * np.linalg.norm(b)
    return it, xs


# flat up to 20480 rows and above 184320, between them clusters of 8 blocks with
# one row a thread up to 61440 and two up to 122880
@pytest.mark.parametrize("n,long_rows", [(1, 0), (31, 0), (33, 0), (257, 0), (20480, 0), (20481, 0), (37889, 0),
                                         (61441, 0), (75777, 0), (122881, 0), (151553, 40), (184321, 0), (40000, 3000),
                                         (303105, 0)])
@pytest.mark.parametrize("guess", [False, True])
def test_solutions(product_lib, n, long_rows, guess):
    check(*spd(n, n, long_rows), seed=n + 1, guess=guess)


def test_threads_share_the_work_space(product_lib):
    systems = [spd(3000 + 500 * k, k) for k in range(4)]
    alone = [check(*s, seed=k) for k, s in enumerate(systems)]
    out = [[] for _ in systems]

    def work(k):
        for _ in range(20):
            out[k].append(check(*systems[k], seed=k))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(len(systems))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for (it, xs), runs in zip(alone, out):
        assert len(runs) == 20
        for i2, x2 in runs:
            assert i2 == it and np.array_equal(x2, xs)
