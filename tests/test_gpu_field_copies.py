"""Device fields in and out of a handle (dglm_get_state, dglm_rhs): the rows of
one array, in any order and at any distance, and separate allocations give the
same values, below and above the size up to which equally spaced rows travel in
one pitched copy (4 MiB per field).  Values are copied, so they are equal bit
for bit."""
import numpy as np
import pytest

from exadglm_b200 import capi, problem as P

pytestmark = pytest.mark.gpu


def _fields(torch, layout, nvar, n):
    if layout == "rows":
        return list(torch.full((nvar, n), -1.0, dtype=torch.float64, device="cuda"))
    if layout == "reversed":
        return list(torch.full((nvar, n), -1.0, dtype=torch.float64, device="cuda"))[::-1]
    if layout == "every other row, odd offset":
        base = torch.full((2 * nvar * n + 1,), -1.0, dtype=torch.float64, device="cuda")[1:]
        return [base[2 * v * n:2 * v * n + n] for v in range(nvar)]
    if layout == "unequal distances":
        base = torch.full((2 * nvar * n,), -1.0, dtype=torch.float64, device="cuda")
        return [base[o * n:o * n + n] for o in (0, 2, 3, 6, 9)]
    return [torch.full((n,), -1.0, dtype=torch.float64, device="cuda") for _ in range(nvar)]


@pytest.mark.parametrize("n", [3, 17])   # 25 KB and 4.7 MB per field
@pytest.mark.parametrize("layout", ["rows", "reversed", "every other row, odd offset",
                                    "unequal distances", "separate"])
def test_field_layouts(layout, n):
    torch = pytest.importorskip("torch")
    p = P.euler_sine(n=n, N=3)
    s = capi.Solver(p)
    s.step(1)
    want = np.asarray(s.get_state()).reshape(p.nvar, -1)
    u = _fields(torch, layout, p.nvar, want.shape[1])
    s.get_state_device([x.data_ptr() for x in u])
    for v in range(p.nvar):
        assert np.array_equal(u[v].cpu().numpy(), want[v])
    ref = torch.empty((p.nvar, want.shape[1]), dtype=torch.float64, device="cuda")
    plain = torch.from_numpy(want).cuda()
    s.rhs_device([x.data_ptr() for x in plain], [x.data_ptr() for x in ref])
    out = _fields(torch, layout, p.nvar, want.shape[1])
    s.rhs_device([x.data_ptr() for x in u], [x.data_ptr() for x in out])
    for v in range(p.nvar):
        assert torch.equal(out[v], ref[v])
