"""The coefficient-class kernels (two launches a step) against the node-slot
kernels (five launches), which use the same arithmetic: every result equal bit
for bit, at row lengths around the 8-slot padding, with each source type, and
on a grid beyond the programmatic-launch limit."""
import numpy as np
import pytest

import tetfit_b200 as tb
from tetfit_b200.cases import FitCase, random_spheres, write_fit_cavity

pytestmark = pytest.mark.gpu


def results(script, steps, state=True, **opts):
    with tb.Discretization(script) as d:
        d.prepare(1, **opts)
        assert d.step(steps - 1) == steps - 1
        out = np.zeros((d.info()["n_probes"], 6))
        assert d.step_io(None, out) == 1
        t, v = d.probes()
        assert not len(v) or np.array_equal(v[-1], out)  # an l2norm output has no probes
        return (v, d.flux(), d.losses()) + (d.state() if state else ()), d.info()["cg_variant"]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n,source", [(2, "h"), (7, "h"), (8, "e"), (9, "j"), (15, "h"), (16, "e"), (23, "h")])
def test_class_steps_equal_node_kernels(tmp_path, product_lib, n, source, precision):
    case = FitCase(n=n, steps=30, spheres=random_spheres(6, seed=n), source_type=source,
                   output_mode="l2norm" if n == 15 else "probepoint")
    script = write_fit_cavity(str(tmp_path), case)
    got, var = results(script, 30, precision=precision)
    ref, node = results(script, 30, precision=precision, fit_variant=1)
    assert var == 5 * 9 and node == 0
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_class_steps_on_a_large_grid(tmp_path, product_lib, precision):
    script = write_fit_cavity(str(tmp_path), FitCase(n=216, steps=8, spheres=random_spheres(20, seed=3)))
    got, _ = results(script, 8, state=False, precision=precision)
    ref, _ = results(script, 8, state=False, precision=precision, fit_variant=1)
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)
