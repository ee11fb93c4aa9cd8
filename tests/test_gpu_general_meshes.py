"""The symmetry-adapted kernels on all that dglm_upload_mesh takes, against a
dense kernel on the same arrays: column-major operators, faces and face points
in any order, neighbours that are any nodes at all (a face's trace from several
elements, from the element itself or from its own tile), metrics, normals and
face factors that belong to no tetrahedron, a velocity of its own at every node.

Tolerance: both sum the same products, at most 3 Np + 4 Nfp per value, in
another order, over values of order one (and factors up to 4 in the sums over
the symmetry): 1e-12 of the largest right-hand side is some 200 units of
rounding of such a sum at N=6.  That holds for a right-hand side, and for a step
where its five stages stay near the state they began with; on a geometry of
random numbers an Euler step takes densities through zero, so there only the
right-hand side is compared."""
import numpy as np
import pytest

from exadglm_b200 import capi
from exadglm_b200 import problem as P

pytestmark = pytest.mark.gpu

CASES = [("euler", N) for N in (3, 4, 5, 6)] + [("advection", N) for N in (2, 3, 4, 5, 6)]


def base(phys, N):
    prob = (P.euler_sine(n=3, N=N, noise=1e-2, seed=N) if phys == "euler"
            else P.advection_gaussian(n=3, N=N, width2=0.05))
    return prob, {k: np.array(v, copy=True) for k, v in prob.datain_arrays().items()}


def as_given(prob, arr, rng):
    pass


def column_major(prob, arr, rng):
    pass


def permuted_faces(prob, arr, rng):
    K, Np = prob.K, prob.Np
    Nfp = arr["Fmask"].size // 4
    order = rng.permutation(4)
    points = [rng.permutation(Nfp) for _ in range(4)]
    flat = np.concatenate([order[f] * Nfp + points[f] for f in range(4)])   # new -> old point
    arr["Fmask"] = arr["Fmask"].reshape(-1)[flat]
    arr["LIFT"] = np.asarray(arr["LIFT"]).reshape(Np, 4 * Nfp)[:, flat]
    arr["vmapP"] = arr["vmapP"].reshape(K, 4 * Nfp)[:, flat]
    for n in ("nx", "ny", "nz", "Fscale"):
        arr[n] = arr[n].reshape(K, 4)[:, order]
    new_of = np.argsort(order)
    vf = arr["vmapF"].reshape(K, 4)[:, order]
    arr["vmapF"] = vf // 4 * 4 + new_of[vf % 4]


def any_neighbours(prob, arr, rng):
    K, Np = prob.K, prob.Np
    shape = np.shape(arr["vmapP"])
    v = rng.integers(0, K * Np, np.size(arr["vmapP"]))
    near = rng.random(v.size) < 0.5   # half of them in the element's own tile of 8
    e = np.repeat(np.arange(K), v.size // K)
    tile = np.minimum(e // 8 * 8 + rng.integers(0, 8, v.size), K - 1)
    v[near] = (tile * Np + rng.integers(0, Np, v.size))[near]
    arr["vmapP"] = v.reshape(shape)
    arr["vmapF"] = rng.integers(0, 4 * K, np.size(arr["vmapF"])).reshape(np.shape(arr["vmapF"]))


def any_geometry(prob, arr, rng):
    for n in ("rx", "ry", "rz", "sx", "sy", "sz", "tx", "ty", "tz", "nx", "ny", "nz"):
        arr[n] = rng.standard_normal(np.shape(arr[n]))
    arr["Fscale"] = rng.uniform(0.1, 10.0, np.shape(arr["Fscale"]))
    if prob.vel is not None:
        prob.vel = rng.standard_normal(np.shape(prob.vel))


@pytest.mark.parametrize("change", [as_given, column_major, permuted_faces, any_neighbours,
                                    any_geometry])
@pytest.mark.parametrize("phys,N", CASES)
def test_rhs_and_step_equal_the_dense_kernel(phys, N, change):
    torch = pytest.importorskip("torch")
    prob, arr = base(phys, N)
    change(prob, arr, np.random.default_rng(10 * N))
    descr = capi.variants(phys, N, "fp64")
    sym = [v for v, d in descr if d.startswith("pipe-dmma-sym")][0]
    dense = [v for v, d in descr if d.startswith("dmma")][0]
    u = torch.from_numpy(np.ascontiguousarray(prob.u0)).cuda()
    out = []
    for v in (sym, dense):
        s = capi.Solver(prob, arrays=arr, variant=v,
                        matrix_order="f" if change is column_major else "c")
        r = torch.empty_like(u)
        s.rhs_device([x.data_ptr() for x in u], [x.data_ptr() for x in r])
        s.step(1)
        out.append((r.cpu().numpy(), s.get_state() - prob.u0.reshape(prob.nvar, -1), s.time()[1]))
        s.close()
    (r0, d0, t0), (r1, d1, t1) = out
    assert np.isfinite(r1).all() and np.abs(r1).max() > 0
    assert np.abs(r0 - r1).max() <= 1e-12 * np.abs(r1).max()
    # the step: the same, over a dt that is the same bit for bit
    assert t0 == t1
    if change is not any_geometry or phys == "advection":
        scale = max(np.abs(d1).max(), np.abs(prob.u0).max())
        assert np.abs(d0 - d1).max() <= 1e-12 * scale
