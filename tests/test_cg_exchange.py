"""The exchange of partial sums in the resident CG kernels: its numbers do not
depend on the iteration limit and may wrap, a wait that can never complete ends
the launch with an error status."""
import os

import numpy as np
import pytest

import tetfit_b200 as tb
from tetfit_b200.cases import TetCase, write_tet_case


@pytest.mark.parametrize("args", [
    dict(blocks=0), dict(blocks=4, cluster=0), dict(blocks=6, cluster=3), dict(blocks=4, cluster=8),
    dict(blocks=32, cluster=32), dict(blocks=66, cluster=2), dict(blocks=4, first=0), dict(blocks=4, rounds=0),
    dict(blocks=4, absent=4), dict(blocks=16, cluster=8, absent=4), dict(blocks=4, timeout_us=0),
    dict(blocks=4, timeout_us=2_000_000),
])
def test_exchange_check_rejects_bad_arguments(product_lib, args):
    with pytest.raises(tb.TetfitError) as e:
        tb.exchange_check(**args)
    assert e.value.code == tb.TF_E_ARG
    assert "tf_exchange_check" in tb.last_thread_error()


@pytest.mark.gpu
@pytest.mark.parametrize("blocks,cluster", [(1, 1), (2, 1), (33, 1), (148, 1), (2, 2), (8, 8), (120, 8), (16, 16)])
@pytest.mark.parametrize("first", [1, 2 ** 31 - 6, 2 ** 32 - 7])
def test_sums_across_the_numbers_range(product_lib, blocks, cluster, first):
    import torch
    blocks = min(blocks, torch.cuda.get_device_properties(0).multi_processor_count // cluster * cluster)
    assert tb.exchange_check(blocks, cluster, first=first, rounds=500)[0] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("blocks,cluster,absent", [(2, 1, 1), (148, 1, 1), (120, 8, 8)])
def test_wait_that_cannot_complete_reports_status(product_lib, blocks, cluster, absent):
    import torch
    blocks = min(blocks, torch.cuda.get_device_properties(0).multi_processor_count // cluster * cluster)
    status, ms = tb.exchange_check(blocks, cluster, rounds=50, absent=absent, timeout_us=20000)
    assert status == 2
    assert 19.0 <= ms < 1000.0
    assert tb.exchange_check(blocks, cluster, rounds=50)[0] == 0  # the context is still usable


# one cluster of 16 blocks, boxes between a few blocks, clusters of 8, boxes on
# 148 blocks, and several simulations in one launch
@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [(9,), (11,), (24,), (28,), (3, 9, 14)])
def test_iteration_limit_leaves_the_solve_alone(tmp_path, product_lib, sizes):
    members = [(write_tet_case(os.path.join(str(tmp_path), f"m{n}"), TetCase(n=n, method="gfdtd", seed=n, steps=40)), 1)
               for n in sizes]

    def run(limit):
        with tb.Batch(members, precision="fp64", cg_maxiter=limit) as b:
            assert b.info(0)["cg_variant"] == 2
            assert b.step(40) == 40
            return [b.state(m) + (b.solver_stats(m)[0],) for m in range(len(members))]

    ref = run(1000)
    assert max(r[3].max() for r in ref) < 1000
    for limit in (2 ** 30, 2 ** 31 - 1):
        for a, r in zip(run(limit), ref):
            for u, v in zip(a, r):
                assert np.array_equal(u, v)
