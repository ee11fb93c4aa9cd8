"""The symmetry-adapted FP64 kernels (variants "pipe-dmma-sym").

On the CPU: the decomposition it computes (projections on the characters of
the four vertex permutations, restated here in numpy from its definition)
against the dense operators, on random fluxes.  Both are sums of at most
3 Np + 4 Nfp products in FP64; the bound, 1e-13 of the sum of the products'
magnitudes, is about 450 units of rounding of that sum (the operators' own
symmetry holds to some 30).

On the GPU, against the oracle (the state bar of the parity tests, 1e-12): tile
remainders, meshes smaller than the grid and several times a block's ring of
buffers; operators without the symmetry, which run on the variant's fallback;
and a change of variant in the middle of a step, where the register changes
its order."""
import numpy as np
import pytest

import oracle
from exadglm_b200 import problem as P
from exadglm_b200.capi import Solver, variants
from exadglm_b200.mesh import Mesh3D, UniformBox
from exadglm_b200.refelem import ref_element

TOL = 1e-12


def rel(a, b):
    return float(np.linalg.norm(np.ravel(a) - np.ravel(b)) / np.linalg.norm(np.ravel(b)))


PHYS = [("euler", N) for N in (3, 4, 5, 6)] + [("advection", N) for N in (2, 3, 4, 5, 6)]


def make(phys, N, cells):
    mesh = Mesh3D(N, UniformBox(*(c + 1 for c in cells)), high_order=False)
    if phys == "euler":
        return P.euler_sine(N=N, noise=1e-3, seed=N, mesh=mesh)
    prob = P.advection_gaussian(N=N, width2=0.05, mesh=mesh)
    # a velocity of its own at every node (tau and the fluxes take it as it is)
    prob.vel = prob.vel * (1 + 0.1 * np.random.default_rng(N).standard_normal(prob.vel.shape))
    return prob


def sym_variant(phys, N):
    return [v for v, d in variants(phys, N, "fp64") if d.startswith("pipe-dmma-sym")][0]


@pytest.mark.parametrize("N", range(1, 9))
def test_decomposition_equals_dense_operators(N):
    ref = ref_element(N)
    lattice = [(N - a - b - c, a, b, c) for c in range(N + 1) for b in range(N + 1 - c)
               for a in range(N + 1 - b - c)]
    index = {q: i for i, q in enumerate(lattice)}
    perm = np.array([[index[tuple(q[i ^ a] for i in range(4))] for q in lattice]
                     for a in range(4)])
    Np, Fmask = len(lattice), np.asarray(ref.Fmask).reshape(4, -1)
    face_of = [[f for f in range(4) if all(lattice[n][v] == 0 for n in Fmask[f])][0]
               for v in range(4)]
    Nfp = Fmask.shape[1]
    pos = [[list(Fmask[face_of[v]]).index(perm[v][n]) for n in Fmask[face_of[0]]]
           for v in range(4)]
    rng = np.random.default_rng(N)
    f, phi = rng.standard_normal((3, Np)), rng.standard_normal((4, Nfp))
    WD, L = [ref.WDr, ref.WDs, ref.WDt], np.asarray(ref.LIFT).reshape(Np, 4, Nfp)
    dense = sum(w @ x for w, x in zip(WD, f)) - np.einsum("ifj,fj->i", L, phi)
    size = sum(abs(w) @ abs(x) for w, x in zip(WD, f)) + np.einsum("ifj,fj->i", abs(L), abs(phi))

    W0 = -(WD[0] + WD[1] + WD[2]) / 4
    W = [W0] + [w + W0 for w in WD]
    W0 = sum(W[v][np.ix_(perm[v], perm[v])] for v in range(4)) / 4
    L0 = sum(L[perm[v]][:, face_of[v]][:, pos[v]] for v in range(4)) / 4
    g = [np.zeros(Np)] + [x + f.sum(0) for x in f]
    y = np.zeros(Np)
    for c in range(4):
        chi = [1 if c == 0 or a in (0, c) else -1 for a in range(4)]
        h = sum(chi[v] * g[v][perm[v]] for v in range(4))
        hF = sum(chi[v] * phi[face_of[v]][pos[v]] for v in range(4))
        z = W0 @ h - L0 @ hF
        y += sum(chi[a] * z[perm[a]] for a in range(4)) / 4
    assert np.all(np.abs(y - dense) <= 1e-13 * size.max()), np.max(np.abs(y - dense) / size.max())


@pytest.mark.gpu
@pytest.mark.parametrize("phys,N", PHYS)
@pytest.mark.parametrize("cells", [(2, 2, 2), (2, 3, 3), (5, 3, 3), (3, 3, 3), (11, 9, 10)])
def test_sizes_match_oracle(phys, N, cells):
    """K = 48, 108, 270, 162 (whole tiles, remainders of 4, 6 and 2 elements)
    and 5,940, several tiles per group."""
    prob = make(phys, N, cells)
    s = Solver(prob, variant=sym_variant(phys, N))
    s.step(2)
    s.sync()
    uo, _, clk, _ = oracle.Oracle(prob).run(2)
    assert rel(s.get_state(), uo) < TOL
    assert abs(s.time()[0] - clk.t) <= 1e-14 * clk.t
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("phys,N", PHYS)
def test_operators_without_the_symmetry(phys, N):
    prob = make(phys, N, (3, 3, 3))
    arr = {k: np.array(v, copy=True) for k, v in prob.datain_arrays().items()}
    arr["WDs"] = arr["WDs"] * (1 + 1e-9 * np.random.default_rng(0).standard_normal(
        np.shape(arr["WDs"])))
    prob.datain_arrays = lambda: arr
    s = Solver(prob, variant=sym_variant(phys, N))
    assert s.variant() == sym_variant(phys, N)
    s.step(3)
    s.sync()
    assert rel(s.get_state(), oracle.Oracle(prob).run(3)[0]) < TOL
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("phys,N", PHYS)
def test_variant_change_between_stages(phys, N):
    """The five stages of a step on two variants in turn give the state of the
    step on one."""
    prob = make(phys, N, (3, 3, 3))
    other = [v for v, d in variants(phys, N, "fp64") if not d.startswith("pipe-dmma-sym")][0]
    one = Solver(prob, variant=sym_variant(phys, N))
    for st in range(5):
        one.stage(st, 1e-3)
    two = Solver(prob, variant=sym_variant(phys, N))
    for st in range(5):
        two.set_variant(other if st % 2 else sym_variant(phys, N))
        two.stage(st, 1e-3)
    assert rel(two.get_state(), one.get_state()) < 1e-14
    one.close()
    two.close()
