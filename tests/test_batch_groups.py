"""A group's CG launch does not depend on groups opened after it (the kernel's
shared memory grows with a group's members)."""
import os

import numpy as np
import pytest

import tetfit_b200 as tb
from tetfit_b200.cases import TetCase, write_tet_case

pytestmark = pytest.mark.gpu


def test_a_smaller_group_opened_later(tmp_path, product_lib):
    small = write_tet_case(os.path.join(str(tmp_path), "s"), TetCase(n=3, method="gfdtd", steps=30))
    large = write_tet_case(os.path.join(str(tmp_path), "l"), TetCase(n=45, method="gfdtd", steps=30))
    opts = dict(precision="fp32")
    with tb.Batch([(small, 1)] * 300, **opts) as b:
        b.step(2)
        with tb.Batch([(large, 1)], **opts) as one:
            one.step(2)
            b.step(2)
            one.step(2)
            assert np.isfinite(b.state(299)[0]).all() and np.isfinite(one.state(0)[0]).all()
