"""The Euler equations are homogeneous: a state scaled by a power of two has the
right-hand side scaled by it, and the kernels' arithmetic (products, sums,
reciprocals) commutes with that scaling bit for bit as long as no intermediate
leaves the range of normal doubles.  Scales up to 2^+-600 are far inside the
range of the states and fluxes themselves, and past that of their squares."""
import numpy as np
import pytest

from exadglm_b200 import capi
from exadglm_b200 import problem as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 3, 4, 5, 6])
@pytest.mark.parametrize("power", [-600, -300, 300, 600])
def test_rhs_of_a_scaled_state(N, power):
    torch = pytest.importorskip("torch")
    prob = P.euler_sine(n=3, N=N, noise=1e-3, seed=N)
    s = capi.Solver(prob)
    u = torch.from_numpy(np.ascontiguousarray(prob.u0)).cuda()
    scale = float(2.0 ** power)
    out = []
    for x in (u, u * scale):
        r = torch.empty_like(x)
        s.rhs_device([v.data_ptr() for v in x], [v.data_ptr() for v in r])
        out.append(r)
    assert torch.equal(out[0] * scale, out[1])
    s.close()
