"""A change of variant of a handle with a state costs its device work, not a
trip of the RK register over the host: the register of the mesh used is 37 MB,
which two host copies and a reordering there take some 100 ms for."""
import time

import pytest

from exadglm_b200 import capi
from exadglm_b200 import problem as P
from exadglm_b200.mesh import Mesh3D, UniformBox

pytestmark = pytest.mark.gpu


def test_change_of_variant_stays_on_the_device():
    prob = P.euler_sine(N=5, mesh=Mesh3D(5, UniformBox(15, 15, 15), high_order=False))
    descr = capi.variants("euler", 5, "fp64")
    sym = [v for v, d in descr if d.startswith("pipe-dmma-sym")][0]
    dense = [v for v, d in descr if not d.startswith("pipe-dmma-sym")][0]
    s = capi.Solver(prob, variant=sym)
    s.step(1)
    s.sync()
    took = []
    for _ in range(5):
        t = time.perf_counter()
        s.set_variant(dense)
        s.set_variant(sym)
        s.sync()
        took.append(time.perf_counter() - t)
    assert min(took) < 0.03, took
    s.close()
