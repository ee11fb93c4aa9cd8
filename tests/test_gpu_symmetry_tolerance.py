"""Operators stand for themselves unless they are symmetric to rounding: one
entry off by 2.5e-14 of the largest (1.4e-14 from the average of its images, a
few times what the rounding of the operators' construction leaves) runs on the
dense variant that the symmetry-adapted one names as its fallback, with its
results bit for bit."""
import numpy as np
import pytest

from exadglm_b200 import capi
from exadglm_b200 import problem as P

pytestmark = pytest.mark.gpu

# the dense variant that stands in, by its description
FALLBACK = {
    ("euler", 3): "pipe-dmma E=16 WN=1 WM=3 threads=352",
    ("euler", 4): "pipe-dmma E=8 WN=1 WM=5 threads=544 smem=195064 ring=2 prod=2 ksplit=3 fused",
    ("euler", 5): "pipe-dmma E=8 WN=5 WM=1 threads=512",
    ("euler", 6): "pipe-dmma E=8 WN=5 WM=2 threads=416",
    ("advection", 2): "dmma E=64 WN=2 WM=2",
    ("advection", 3): "pipe-dmma E=32 WN=1 WM=3 threads=448",
    ("advection", 4): "pipe-dmma E=32 WN=1 WM=5",
    ("advection", 5): "pipe-dmma E=16 WN=1 WM=7",
    ("advection", 6): "pipe-dmma E=8 WN=1 WM=11 threads=448",
}


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
    dense = [v for v, d in capi.variants(phys, N, "fp64") if d.startswith(FALLBACK[phys, N])]
    assert len(dense) == 1 and np.array_equal(got, run(entry, dense[0]))
