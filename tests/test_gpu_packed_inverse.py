"""Coarsest levels large enough for the packed symmetric product (2304 DOFs, a
ragged last tile): the V-cycle against the one that reads the inverse whole
(the persistent coarse kernel), and batched solves against single ones over
more right-hand sides than one pass over the tiles takes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[False, True])
def solver(request):
    from top_gpu_on_matlab_b200.fea import Mesh, Solver
    m = Mesh(np.ones((56, 88, 56), bool), control=20000)
    assert 3 * m.info()[-1]["numNodes"] == 2304
    ny, nx, nz = 56, 88, 56
    g = np.arange((ny + 1) * (nx + 1) * (nz + 1))
    X = g // (ny + 1) % (nx + 1)
    fix = np.column_stack([g[X == 0] + 1, np.ones((int((X == 0).sum()), 3))]).astype(float)
    end = g[X == nx] + 1
    r = np.random.default_rng(1)
    m.apply_bc(fix, [np.column_stack([end, r.standard_normal((len(end), 3)) / len(end)]) for _ in range(5)])
    s = Solver(m, E0=1.0, Emin=1e-9, penal=3.0, tol=1e-6, maxIT=200, omega=0.6, mixed=request.param)
    s.set_density(torch.from_numpy(0.4 + 0.6 * r.random(s.num_design)).cuda())
    s.assemble()
    return s


def test_vcycle_equals_the_whole_inverse(solver):
    u = torch.from_numpy(np.random.default_rng(2).standard_normal(solver.numDOFs)).cuda()
    z = solver.vcycle(u)
    solver.set_coarse_persistent(1)
    try:
        w = solver.vcycle(u)                    # switched on an assembled solver
        solver.assemble()
        w2 = solver.vcycle(u)
    finally:
        solver.set_coarse_persistent(0)
    assert torch.equal(w, w2)
    # the same sums of n = 2304 terms in another order: n eps = 5e-13, in single one rounding of x besides
    tol = 1e-6 if solver.params.precision else 1e-11
    assert float((z - w).abs().max()) < tol * float(w.abs().max())


def test_batched_equals_single(solver):
    U, its, _ = solver.pcg_all()
    n = solver.numDOFs
    for k in range(5):
        Uk, ik, _ = solver.pcg(k)
        assert ik == its[k] and torch.equal(U[k * n:(k + 1) * n], Uk)
