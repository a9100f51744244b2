"""The condensed tail on a coarsest level that is kept as packed tiles: separate
bodies, each as small as a coarsest cell, so that the level above the coarsest
has few enough DOFs for the tail and the coarsest more than the packed form
asks for (37,500, 2400 and 2400).  The tail against the launched steps in both
precisions, formed at assembly and switched on afterwards."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a - b).abs().max() / b.abs().max())


@pytest.fixture(scope="module")
def mesh():
    from top_gpu_on_matlab_b200.fea import Mesh
    mask = np.zeros((160, 8, 160), bool)
    for y in range(0, 160, 16):
        for z in range(0, 160, 16):
            mask[y:y + 4, :4, z:z + 4] = True
    m = Mesh(mask, control=400)
    lv = m.info()
    assert [3 * q["numNodes"] for q in lv] == [37500, 2400, 2400]
    NY, NX = lv[0]["resY"] + 1, lv[0]["resX"] + 1
    fwd = m.get(0, "nodMapForward")
    act = np.flatnonzero(fwd)
    X = act // NY % NX
    fix, end = fwd[act[X == 0]], fwd[act[X == 4]]       # every body is held at x = 0 and loaded at x = 4
    load = np.random.default_rng(1).standard_normal((len(end), 3)) / len(end)
    m.apply_bc(np.column_stack([fix, np.ones((len(fix), 3))]).astype(float), [np.column_stack([end, load])])
    return m


def _solver(mesh, mixed):
    from top_gpu_on_matlab_b200.fea import Solver
    s = Solver(mesh, E0=1.0, Emin=1e-9, penal=3.0, tol=1e-8, maxIT=400, omega=0.6, mixed=mixed)
    s.set_density(torch.from_numpy(0.4 + 0.6 * np.random.default_rng(2).random(s.num_design)).cuda())
    return s


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("when", ["at assembly", "afterwards"])
def test_tail_on_a_packed_coarsest_level(mesh, mixed, when):
    s = _solver(mesh, mixed)
    assert s.set_tail_operator(when == "at assembly") == (1 if when == "at assembly" else 0)
    s.assemble()
    r = torch.from_numpy(np.random.default_rng(3).standard_normal(s.numDOFs)).cuda()
    assert s.set_tail_operator(False) == 0
    z0 = s.vcycle(r)
    if when == "at assembly":
        s.set_tail_operator(True)
        s.assemble()
    assert s.set_tail_operator(True) == 1
    # the same operator as sums of 2400 terms in another order (n eps = 5e-13); in single one rounding of M and x besides
    assert _rel(s.vcycle(r), z0) < (1e-5 if mixed else 1e-11)


def test_mixed_uses_the_tail_by_default(mesh):
    s = _solver(mesh, True)
    s.assemble()
    r = torch.from_numpy(np.random.default_rng(4).standard_normal(s.numDOFs)).cuda()
    z1 = s.vcycle(r)
    assert s.set_tail_operator(None) == 1 and s.set_tail_operator(False) == 0
    assert _rel(z1, s.vcycle(r)) < 1e-5
