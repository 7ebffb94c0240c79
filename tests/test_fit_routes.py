"""Routes of a FIT step against the node-slot kernels bit for bit: scenes of more
coefficient classes than the class kernels' tables hold, on a grid that the march
kernels take and on one that the autotuner measures; the class kernels on both
sides of the limit of their programmatic launches."""
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import tetfit_b200 as tb
from tetfit_b200.cases import FitCase, Sphere, random_spheres, write_fit_cavity

pytestmark = pytest.mark.gpu


def write_many_classes(directory, n, steps, block=36, materials=250):
    """A cavity whose first block^3 cells each have one of 250 materials at
    random: about 140,000 different edges and 90,000 different faces."""
    r = np.random.default_rng(9)
    table = [Sphere((9.0, 9.0, 9.0), 0.1, float(e), float(s))
             for e, s in zip(r.uniform(1, 6, materials), r.uniform(0, 0.02, materials))]
    script = write_fit_cavity(directory, FitCase(n=n, steps=steps, spheres=table))
    labels = r.integers(1, materials + 1, block ** 3)
    h = 1.0 / n
    lines = []
    for q, m in enumerate(labels):
        c = [((q // block ** a) % block + 0.5) * h for a in range(3)]
        lines += [f"DEFINE solid {q + 1}", f"   SET material {m}", "   SET type sphere",
                  "   SET center {%r,%r,%r}" % tuple(c), f"   SET radius {0.3 * h!r}", f"END solid {q + 1}"]
    q = len(labels) + 1
    lines += [f"DEFINE solid {q}", f"   SET material {materials + 1}", "   SET type box", "   SET corner {0,0,0}",
              "   SET size {1,1,1}", f"END solid {q}"]
    with open(os.path.join(directory, "cavity_solids.txt"), "w") as f:
        f.write("\n".join(lines) + "\n")
    return script


def results(script, steps, state, **opts):
    with tb.Discretization(script) as d:
        d.prepare(1, **opts)
        assert d.step(steps) == steps
        return (d.probes()[1], d.flux()) + (d.state() if state else ()), d.info()["cg_variant"]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n,steps", [(36, 40), (216, 16)])
def test_more_classes_than_the_tables_hold(tmp_path, product_lib, n, steps, precision):
    script = write_many_classes(str(tmp_path), n, steps)
    got, variant = results(script, steps, n < 100, precision=precision)
    ref, _ = results(script, steps, n < 100, precision=precision, fit_variant=1)
    assert variant == 2 * 9 if n < 100 else (variant % 8 != 5 and variant // 8 != 5)
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)


# launches of up to 2,048 blocks are programmatic, in FP64 to about 97^3 cells (the
# two runs' host set-up, most of the test's time, goes side by side)
@pytest.mark.parametrize("n", [95, 100])
def test_class_steps_on_both_sides_of_the_programmatic_limit(tmp_path, product_lib, n):
    script = write_fit_cavity(str(tmp_path), FitCase(n=n, steps=20, spheres=random_spheres(20, seed=n)))
    with ThreadPoolExecutor(2) as pool:
        (got, variant), (ref, node) = pool.map(lambda v: results(script, 20, True, fit_variant=v), (0, 1))
    assert variant == 5 * 9 and node == 0
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)
