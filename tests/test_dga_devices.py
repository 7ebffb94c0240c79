"""A dga state is read through an export kernel on the simulation's device,
whatever device the calling thread has current (needs two GPUs)."""
import threading

import numpy as np
import pytest

import tetfit_b200 as tb
from tetfit_b200.cases import TetCase, write_tet_case


@pytest.mark.gpu
def test_state_with_another_device_current(tmp_path, product_lib):
    import torch
    if torch.cuda.device_count() < 2:
        pytest.skip("one device")
    script = write_tet_case(str(tmp_path), TetCase(n=4, method="dga", steps=20))
    sims = []
    for device in (0, 1):
        d = tb.Discretization(script)
        d.prepare(1, precision="fp64", device=device)  # leaves its device current
        d.step(20)
        sims.append(d)
    states = [d.state() for d in sims]
    torch.cuda.set_device(0)
    sims[1].state()
    assert torch.cuda.current_device() == 0
    fresh = [None]
    t = threading.Thread(target=lambda: fresh.__setitem__(0, sims[1].state()))  # device 0 current
    t.start()
    t.join()
    assert fresh[0] is not None
    for a, b, c in zip(*states, fresh[0]):
        assert np.array_equal(a, b) and np.array_equal(a, c)
