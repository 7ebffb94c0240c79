"""The dga device numbering (chunks of 4096 rows by stencil, SELL-32) and its
captured step: states go in and out in the reference's numbering, captured and
single steps give the same bits, at sizes below, around and above a chunk and
with every edge class."""
import numpy as np
import pytest

import oracle
import tetfit_b200 as tb
from tetfit_b200.cases import TetCase, write_tet_case

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("fp32", 1e-5)])
@pytest.mark.parametrize("n,kw", [(2, {}), (8, dict(split_x=True, eps=(1.0, 2.5))), (9, dict(source_type="e")),
                                  (6, dict(split_x=True, eps=(1.0, 2.0), sigma=(0.0, 0.02))),
                                  (5, dict(chi=(3e3,)))])
def test_captured_steps_and_states(tmp_path, product_lib, oracle_lib, n, kw, precision, tol):
    if precision == "fp32" and ("sigma" in kw or "chi" in kw):
        tol = 1e-4  # the bound of the lossy parity tests for F and the flux
    script = write_tet_case(str(tmp_path), TetCase(n=n, method="dga", steps=45, **kw))
    o = oracle.TetOracle(script)
    o.step(o.n_steps)
    _, vo, _, _ = o.probes()
    ref = o.state() + (vo, o.flux())
    runs = []
    for graph in (0, 1, 7):
        with tb.Discretization(script) as d:
            d.prepare(1, precision=precision, graph_steps=graph)
            for k in (1, 20, 3, 1000):
                d.step(k)
            runs.append(d.state() + (d.probes()[1], d.flux()))
            if graph == 0 and "sigma" not in kw:
                U, B, F = runs[-1][:3]
                d.set_state(U, F)
                again = d.state()
                assert np.array_equal(again[0], U) and np.array_equal(again[2], F)
    for a, r in zip(runs[0], ref):
        assert rel(a, r) <= tol
    for other in runs[1:]:
        for a, b in zip(runs[0], other):
            assert np.array_equal(a, b)
