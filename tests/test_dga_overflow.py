"""An infinity in a dga state reaches the values that depend on it and no
others become NaN: the padding of the 32-row slices reads nothing that is not
zero.  Which values turn infinite or NaN follows from the operators' rows."""
import numpy as np
import pytest

import oracle
import tetfit_b200 as tb
from tetfit_b200.cases import TetCase, write_tet_case

pytestmark = pytest.mark.gpu


def rows_of(matrix, x):
    ptr, col, val = matrix
    row = np.repeat(np.arange(len(ptr) - 1), np.diff(ptr.astype(np.int64)))
    y = np.zeros(len(ptr) - 1)
    np.add.at(y, row, val * x[col])
    return y


def transposed(matrix, x, n):
    ptr, col, val = matrix
    row = np.repeat(np.arange(len(ptr) - 1), np.diff(ptr.astype(np.int64)))
    y = np.zeros(n)
    np.add.at(y, col, val * x[row])
    return y


def same_kind(a, r):
    return (np.array_equal(np.isnan(a), np.isnan(r)) and np.array_equal(np.isposinf(a), np.isposinf(r)) and
            np.array_equal(np.isneginf(a), np.isneginf(r)))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_infinity_stays_in_its_rows(tmp_path, product_lib, oracle_lib, precision):
    script = write_tet_case(str(tmp_path), TetCase(n=4, method="dga", steps=200))
    o = oracle.TetOracle(script)
    C, N, H = (o.matrix(w) for w in "CNH")
    live = np.diff(H[0].astype(np.int64)) > 0
    rng = np.random.default_rng(3)
    with tb.Discretization(script) as d, np.errstate(invalid="ignore"):
        d.prepare(1, precision=precision)
        for e in rng.choice(np.flatnonzero(live), 20, replace=False):
            U = np.zeros(o.nE)
            U[e] = np.inf
            d.set_state(U, np.zeros(o.nF))
            d.step(1)
            Un, _, F = d.state()
            assert same_kind(F, -rows_of(N, rows_of(C, Un)))
        for f in rng.choice(o.nF, 20, replace=False):
            F = np.zeros(o.nF)
            F[f] = np.inf
            d.set_state(np.zeros(o.nE), F)
            d.step(1)
            assert same_kind(d.state()[0][live], rows_of(H, transposed(C, F, o.nE))[live])
