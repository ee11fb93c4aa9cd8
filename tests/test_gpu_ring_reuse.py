"""The symmetry-adapted kernels where their buffers go round: meshes sized by
the number of SMs so that a block of the Euler kernel takes more than twice its
ring of tiles, and every warp of the advection and batch kernels at least three
(prefetch, both parities of its two buffers, a store before a refill), with a
ragged last tile.  Against the oracle, at the state bar of the parity tests."""
import numpy as np
import pytest

import oracle
from exadglm_b200 import capi
from exadglm_b200 import problem as P
from exadglm_b200.mesh import Mesh3D, UniformBox

pytestmark = pytest.mark.gpu

TOL = 1e-12

# tiles of 8 elements per block: the Euler ring (2 NB + 1), advection 3 per warp
EULER = {3: 17, 4: 13, 5: 7, 6: 5}
ADVECTION = {2: 48, 3: 72, 4: 48, 5: 48, 6: 24}


def rel(a, b):
    return float(np.linalg.norm(np.ravel(a) - np.ravel(b)) / np.linalg.norm(np.ravel(b)))


def cells(K):
    """The smallest box of nearly equal sides with at least K tetrahedra, not a
    whole number of tiles."""
    n = 2
    while True:
        for c in ((n, n, n), (n, n, n + 1), (n, n + 1, n + 1), (n, n + 1, n + 2)):
            k = 6 * c[0] * c[1] * c[2]
            if k >= K and k % 8:
                return c
        n += 1


@pytest.mark.parametrize("phys,N", [("euler", N) for N in EULER] +
                         [("advection", N) for N in ADVECTION])
def test_many_tiles_per_warp(phys, N):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    per = (EULER if phys == "euler" else ADVECTION)[N]
    c = cells(8 * sms * per)
    mesh = Mesh3D(N, UniformBox(*(x + 1 for x in c)), high_order=False)
    prob = (P.euler_sine(N=N, noise=1e-3, seed=N, mesh=mesh) if phys == "euler"
            else P.advection_gaussian(N=N, width2=0.05, mesh=mesh))
    v = [v for v, d in capi.variants(phys, N, "fp64") if d.startswith("pipe-dmma-sym")][0]
    s = capi.Solver(prob, variant=v)
    s.step(2)
    s.sync()
    uo, _, clk, _ = oracle.Oracle(prob).run(2)
    assert rel(s.get_state(), uo) < TOL
    assert abs(s.time()[0] - clk.t) <= 1e-14 * clk.t
    s.close()


def batch_problems(sizes):
    return [P.advection_gaussian(n=n, N=N, width2=0.02 + 0.01 * N, v=(0.3, -0.5, 0.1 * N))
            for n, N in sizes]


def test_batch_with_many_tiles_per_warp():
    """Cut by cost, a block's stretch of N=6 tiles (the dearest) is 30 tiles for
    its 8 warps; the other orders' are longer."""
    probs = batch_problems([(13, 2), (13, 3), (13, 4), (13, 5), (13, 6), (11, 6)])
    b = capi.BatchSolver(probs)
    b.step(2)
    b.sync()
    for i, p in enumerate(probs):
        assert p.K % 8
        assert rel(b.get_state(i), oracle.Oracle(p).run(2)[0]) < TOL
    b.close()


def test_batch_of_operators_without_the_symmetry():
    """One order's operators are enough for the whole batch to run on the dense
    kernel."""
    probs = batch_problems([(4, 2), (3, 3), (5, 4), (3, 5), (3, 6), (4, 4)])
    for p in probs:
        arr = {k: np.array(v, copy=True) for k, v in p.datain_arrays().items()}
        if p.N == 4:
            arr["WDs"] = arr["WDs"] * (1 + 1e-9 * np.random.default_rng(0).standard_normal(
                np.shape(arr["WDs"])))
        p.datain_arrays = lambda arr=arr: arr
    b = capi.BatchSolver(probs)
    b.set_wait_limit(1)   # (no bounded waits there)
    b.step(3)
    b.sync()
    for i, p in enumerate(probs):
        assert rel(b.get_state(i), oracle.Oracle(p).run(3)[0]) < TOL
    b.close()
