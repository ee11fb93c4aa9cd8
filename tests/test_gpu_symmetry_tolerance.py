"""Operators stand for themselves unless they are symmetric to rounding: one
entry off by 2.5e-14 of the largest (1.4e-14 from the average of its images, a
few times what the rounding of the operators' construction leaves) runs on the
dense kernels, with their results bit for bit."""
import numpy as np
import pytest

from exadglm_b200 import capi
from exadglm_b200 import problem as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("phys,N", [("euler", N) for N in (3, 4, 5, 6)] +
                         [("advection", N) for N in (2, 3, 4, 5, 6)])
def test_operators_off_by_more_than_rounding(phys, N):
    prob = (P.euler_sine(n=3, N=N, noise=1e-3, seed=N) if phys == "euler"
            else P.advection_gaussian(n=3, N=N, width2=0.05))
    sym = [v for v, d in capi.variants(phys, N, "fp64") if d.startswith("pipe-dmma-sym")][0]

    def run(entry, variant):
        arr = {k: np.array(v, copy=True) for k, v in prob.datain_arrays().items()}
        arr["WDs"].reshape(-1)[entry] += 2.5e-14 * np.abs(arr["WDs"]).max()
        s = capi.Solver(prob, arrays=arr, variant=variant)
        s.step(2)
        out = s.get_state()
        s.close()
        return out

    entry = prob.Np + 2   # (row 1, column 2)
    got = run(entry, sym)
    dense = [v for v, d in capi.variants(phys, N, "fp64") if not d.startswith("pipe-dmma-sym")]
    assert any(np.array_equal(got, run(entry, v)) for v in dense)
