"""Bounded waits of the FP64 stage kernels, kernel by kernel: with a bound of
one cycle a step's waits run out, the step is reported, and the same handle
steps as before after a new state.  (The host shortens the bound; every warp
waits for its own copies with the normal one before it leaves.)"""
import numpy as np
import pytest

import oracle
from exadglm_b200 import capi
from exadglm_b200 import problem as P

pytestmark = pytest.mark.gpu

TOL = 1e-12   # the state bar of the parity tests


def rel(a, b):
    return float(np.linalg.norm(np.ravel(a) - np.ravel(b)) / np.linalg.norm(np.ravel(b)))


def problem(phys, N):
    return (P.euler_sine(n=6, N=N, noise=1e-3, seed=4) if phys == "euler"
            else P.advection_gaussian(n=6, N=N, width2=0.05))


def expire_and_recover(prob, variant):
    ref = oracle.Oracle(prob).run(2)[0]
    s = capi.Solver(prob, variant=variant)
    s.set_wait_limit(1)
    s.step(1)
    with pytest.raises(capi.DglmError, match="bounded wait"):
        s.sync()
    s.set_wait_limit(0)
    s.set_state(prob.u0)
    s.step(2)
    s.sync()
    assert rel(s.get_state(), ref) < TOL
    s.close()


@pytest.mark.parametrize("phys,N", [("euler", N) for N in (3, 4, 5, 6)] +
                         [("advection", N) for N in (2, 3, 4, 5, 6)])
def test_symmetry_adapted_kernels(phys, N):
    v = [v for v, d in capi.variants(phys, N, "fp64") if d.startswith("pipe-dmma-sym")][0]
    expire_and_recover(problem(phys, N), v)


@pytest.mark.parametrize("phys,N", [("euler", 3), ("euler", 4), ("euler", 5), ("advection", 3)])
def test_dense_pipelined_kernels(phys, N):
    v = [v for v, d in capi.variants(phys, N, "fp64") if d.startswith("pipe-dmma E=")][0]
    expire_and_recover(problem(phys, N), v)


def test_batch_kernel():
    """One instance per order: every order's tiles wait.  The states of a batch
    whose wait ran out stay invalid; a new batch steps as before."""
    probs = [P.advection_gaussian(n=4, N=N, width2=0.05) for N in (2, 3, 4, 5, 6)]
    b = capi.BatchSolver(probs)
    b.set_wait_limit(1)
    b.step(1)
    for _ in range(2):
        with pytest.raises(capi.DglmError, match="bounded wait"):
            b.sync()
    b.close()
    b = capi.BatchSolver(probs)
    b.step(2)
    b.sync()
    for i, p in enumerate(probs):
        assert rel(b.get_state(i), oracle.Oracle(p).run(2)[0]) < TOL
    b.close()


def test_batch_states_and_times_are_refused_after_expiry():
    """Without a sync in between, too: a caller may step and take the state."""
    probs = [P.advection_gaussian(n=3, N=N, width2=0.05) for N in (3, 5)]
    for take in (lambda b: b.get_state(1), lambda b: b.time(0)):
        b = capi.BatchSolver(probs)
        b.step(1)
        take(b)   # read once: the next step's expiry is seen all the same
        b.set_wait_limit(1)
        b.step(1)
        with pytest.raises(capi.DglmError, match="bounded wait"):
            take(b)
        b.close()
