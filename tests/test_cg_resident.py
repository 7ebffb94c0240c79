"""The resident CG (one block an SM, rows in registers, part of A in shared
memory) against the general CG kernel: members small enough for it alone, then
again in one batch with a member that makes the group too large for it.  Sizes
from a few blocks to several rows a thread with part of A streamed."""
import os
import threading

import numpy as np
import pytest

import tetfit_b200 as tb
from tetfit_b200.cases import TetCase, write_tet_case

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def collect(members, count, steps, **opts):
    with tb.Batch(members, **opts) as b:
        variant = b.info(0)["cg_variant"]
        assert b.step(steps) == steps
        return variant, [(b.state(m), b.probes(m)[1], b.flux(m), b.solver_stats(m)[0]) for m in range(count)]


@pytest.mark.parametrize("precision,warm", [("fp64", "previous"), ("fp32", "extrapolate"), ("fp32", "learned")])
def test_resident_equals_general(tmp_path, product_lib, precision, warm):
    steps = 30 if warm == "learned" else 12
    tol = 1e-13 if precision == "fp64" else 1e-8

    def case(i, n, method="gfdtd"):
        c = TetCase(n=n, method=method, split_x=True, eps=(1.0 + 0.2 * i, 2.5), seed=50 + i, steps=40, tolerance=tol)
        return (write_tet_case(os.path.join(str(tmp_path), f"m{i}"), c), 1)

    # 2^3: one slice in a cluster of 16 blocks; 8^3: a few blocks; 17^3 and 21^3:
    # one and two rows a thread; 36^3: five, part of A streamed in FP64; 24^3 and
    # 32^3: clusters of 8 (32^3 in FP32 alone); fem: 19-entry rows
    groups = [[case(0, 2)], [case(9, 9)], [case(10, 24)], [case(11, 32)], [case(1, 3), case(2, 8), case(3, 5, "fem")], [case(4, 17), case(5, 21)], [case(6, 36)],
              [case(7, 15, "fem")]]
    big = case(8, 48)
    opts = dict(precision=precision, warm_start=warm, cg_criterion="rhs", learn_steps=15)
    for members in groups:
        variant, got = collect(members, len(members), steps, **opts)
        assert variant == 2
        general, ref = collect(members + [big], len(members), steps, **opts)
        assert general in (0, 1)
        for (gs, gp, gf, gi), (rs, rp, rf, ri) in zip(got, ref):
            # the CGs differ in the order of their sums; the learned network
            # also trains on other samples
            assert np.abs(gi - ri).max() <= (3 if warm == "learned" else 1)
            bound = 1e-10 if precision == "fp64" else 1e-5
            for a, r in zip(gs + (gp, gf), rs + (rp, rf)):
                assert rel(a, r) <= bound


def test_simulations_in_threads(tmp_path, product_lib):
    """One cluster of 16, clusters of 8 and flat boxes on 148 blocks at once,
    each from its own thread: the sums have a fixed order, so every state is
    the one of a run alone, bit for bit."""
    scripts = [write_tet_case(os.path.join(str(tmp_path), f"t{n}"), TetCase(n=n, method="gfdtd", seed=n, steps=80))
               for n in (9, 24, 27)]

    def run(script):
        with tb.Discretization(script) as d:
            d.prepare(1, precision="fp64")
            assert d.step(60) == 60
            return d.state() + (d.solver_stats()[0],)

    alone = [run(s) for s in scripts]
    got = [None] * len(scripts)

    def work(k):
        got[k] = run(scripts[k])

    ts = [threading.Thread(target=work, args=(k,)) for k in range(len(scripts))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for a, g in zip(alone, got):
        assert g is not None
        for u, v in zip(a, g):
            assert np.array_equal(u, v)
