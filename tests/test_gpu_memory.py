"""Device memory of FP64 handles: the record of the symmetry-adapted kernels is
held only by handles that run them, and a handle gives it up (running on the
dense fallback from then on) rather than fail where memory is short.

The memory of the GPU is taken up by one tensor that leaves what the handle
needs without the record and SLACK more (allocation granules and the kernels'
code); the record of the mesh used is 234 MB."""
import contextlib

import numpy as np
import pytest

from exadglm_b200 import capi
from exadglm_b200 import problem as P
from exadglm_b200.mesh import Mesh3D, UniformBox

pytestmark = pytest.mark.gpu

SLACK = 96 << 20


def sym_variant(phys, N):
    return [v for v, d in capi.variants(phys, N, "fp64") if d.startswith("pipe-dmma-sym")][0]


def solver(prob, variant):
    return capi.Solver(prob, variant=variant)


@contextlib.contextmanager
def memory_left(leave):
    """All device memory but `leave` bytes is taken."""
    torch = pytest.importorskip("torch")
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")
    yield
    del hold
    torch.cuda.empty_cache()


@pytest.mark.parametrize("phys,N", [("euler", 1), ("euler", 2), ("euler", 4), ("euler", 7),
                                    ("advection", 2), ("advection", 5)])
def test_only_handles_that_run_the_symmetry_adapted_kernels_hold_a_record(phys, N):
    n = 3
    prob = P.euler_sine(n=n, N=N) if phys == "euler" else P.advection_gaussian(n=n, N=N)
    Np, Nfp, nvar, Kp = prob.Np, (N + 1) * (N + 2) // 2, prob.nvar, -(-prob.K // 64) * 64
    fields = 3 * nvar + (3 if phys == "advection" else 0)
    # fields, metrics, normals, Fscale, tau, maxv, and the maps
    mesh = Kp * (8 * (fields * Np + 9 + 12 + 3 * 4) + 4 * (4 * Nfp + 4))
    rest = 65536 * 8 + 4 * 4 * Nfp + 4096   # dt history, Fmask, scalars
    dense = [v for v, d in capi.variants(phys, N, "fp64") if not d.startswith("pipe-dmma-sym")][0]
    operators = 8 * 4 * (-(-Np // 8) * 8 + 8) * (3 * Np + 4 * Nfp + 32)   # any layout
    s = solver(prob, -1)
    has = N in ((3, 4, 5, 6) if phys == "euler" else (2, 3, 4, 5, 6))
    s.set_variant(dense)
    assert s.device_bytes() <= mesh + rest + operators
    if has:
        lean = s.device_bytes()
        s.set_variant(sym_variant(phys, N))
        assert s.device_bytes() > lean
        s.set_variant(dense)
        assert s.device_bytes() == lean
    s.close()


@pytest.fixture(scope="module")
def big():
    mesh = Mesh3D(5, UniformBox(26, 26, 26), high_order=False)
    prob = P.advection_gaussian(N=5, width2=0.05, mesh=mesh)
    dense = [v for v, d in capi.variants("advection", 5, "fp64")
             if d.startswith("pipe-dmma E=16")][0]
    s = solver(prob, dense)   # the fallback of the symmetry-adapted variant
    lean = s.device_bytes()
    s.step(2)
    want = s.get_state()
    s.close()
    return prob, lean, want


def test_no_memory_for_the_record(big):
    prob, lean, want = big
    with memory_left(lean + SLACK):
        s = solver(prob, sym_variant("advection", 5))
    assert s.device_bytes() == lean
    s.step(2)
    assert np.array_equal(s.get_state(), want)
    s.close()


def test_record_given_back_for_a_later_allocation(big):
    """The ensemble's four state buffers (168 MB) do not fit beside it."""
    prob, lean, want = big
    s = solver(prob, sym_variant("advection", 5))
    assert s.device_bytes() > lean + 2 * SLACK
    s.step(1)
    s.sync()
    with memory_left(SLACK):
        out = s.run_ensemble([prob.u0], 2)[0]
    assert np.array_equal(out, want)
    assert s.device_bytes() < lean + 4 * 8 * prob.K * prob.Np + (1 << 20)
    s.close()


def test_right_hand_side_without_memory_for_its_scratch(big):
    """Half of the scratch would fit: each call is refused, and the first one
    with the memory back works."""
    torch = pytest.importorskip("torch")
    prob, lean, _ = big
    dense = [v for v, d in capi.variants("advection", 5, "fp64")
             if d.startswith("pipe-dmma E=16")][0]
    s = solver(prob, dense)
    u = torch.from_numpy(prob.u0.copy()).cuda()
    out, want = torch.zeros_like(u), torch.zeros_like(u)

    def rhs(r):
        s.rhs_device([u.data_ptr()], [r.data_ptr()])

    with memory_left(64 << 20):
        for _ in range(2):
            with pytest.raises(capi.DglmError) as e:
                rhs(out)
            assert e.value.status == capi.ERR_NOMEM
    assert s.device_bytes() == lean
    rhs(out)
    fresh = solver(prob, dense)
    fresh.rhs_device([u.data_ptr()], [want.data_ptr()])
    assert torch.equal(out, want) and float(out.abs().max()) > 0
    s.close()
    fresh.close()


def test_record_given_back_between_two_stages():
    """Euler N=4, K=196,608: the element record is 41 MB, and the right-hand side's
    scratch (563 MB) is asked for after the first of five stages, with 24 MB less
    than it needs.  The other stages run on the fallback, from the register as
    the first left it: the state of five stages on one kernel, to rounding."""
    torch = pytest.importorskip("torch")
    prob = P.euler_sine(n=32, N=4)
    variant = sym_variant("euler", 4)
    scratch = 8 * (2 * 5 * 35 + 2 * 4) * prob.K
    states = []
    for squeeze in (False, True):
        s = solver(prob, variant)
        s.step(1)   # wave speeds and tau for the stages
        dt = s.time()[1]
        s.stage(0, dt)
        if squeeze:
            u = torch.from_numpy(prob.u0.copy()).cuda()
            r = torch.empty_like(u)
            before = s.device_bytes()
            with memory_left(scratch - (24 << 20)):
                s.rhs_device([x.data_ptr() for x in u], [x.data_ptr() for x in r])
            assert s.device_bytes() - before < scratch - (32 << 20)   # the record is gone
        for st in range(1, 5):
            s.stage(st, dt)
        states.append(s.get_state())
        s.close()
    a, b = states
    assert np.linalg.norm(a - b) <= 1e-14 * np.linalg.norm(b)


def test_batch_without_memory_for_the_symmetry_adapted_path():
    """Its lists and records are 135 MB of the batch used.  (The two paths'
    sums differ in their order: 1e-13 is the batch tests' bar.)"""
    mesh = Mesh3D(6, UniformBox(25, 25, 25), high_order=False)
    probs = [P.advection_gaussian(N=6, width2=w, mesh=mesh) for w in (0.05, 0.06, 0.07)]

    def run():
        b = capi.BatchSolver(probs)
        b.step(2)
        out = [b.get_state(i) for i in range(len(probs))]
        nbytes = b.device_bytes()
        b.close()
        return out, nbytes

    want, full = run()
    K, Np, Nfp = probs[0].K, 84, 28
    dense = 3 * K * (8 * (3 * Np + 25) + 16 * Nfp)   # states, register, geometry, vmapP
    assert full > dense + SLACK
    with memory_left(dense + SLACK):
        got, lean = run()
    assert lean < dense + (8 << 20)
    for a, b in zip(got, want):
        assert np.linalg.norm(a - b) <= 1e-13 * np.linalg.norm(b)
