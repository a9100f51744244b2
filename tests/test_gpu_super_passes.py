"""Which form of the packed product super elements take at level 0: one launch
where the one-pass kernel's CTAs are one resident wave (a product, or in
single a batch of them), two from there on; each with the result of the other."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _solver(shape, mixed, loads=1):
    from top_gpu_on_matlab_b200.fea import Mesh, Solver
    ny, nx, nz = shape
    m = Mesh(np.ones(shape, bool), control=20000, super_element=1)
    g = np.arange((ny + 1) * (nx + 1) * (nz + 1))
    X = g // (ny + 1) % (nx + 1)
    r = np.random.default_rng(1)
    fix, end = g[X == 0] + 1, g[X == nx] + 1
    m.apply_bc(np.column_stack([fix, np.ones((len(fix), 3))]).astype(float),
               [np.column_stack([end, r.standard_normal((len(end), 3)) / len(end)]) for _ in range(loads)])
    s = Solver(m, E0=1.0, Emin=1e-9, penal=3.0, tol=1e-8, maxIT=800, omega=0.6, mixed=mixed)
    s.set_density(torch.from_numpy(0.3 + 0.7 * r.random(s.num_design)).cuda())
    s.assemble()
    return s


def _launches(s, call):
    n = s.launches
    out = call()
    return s.launches - n, out


# one-pass CTAs a right-hand side (20 slots in y, 32 a CTA): 527 and 612 around one wave of 4 x 148, 63 the smallest
@pytest.mark.parametrize("shape,passes", [((3, 5, 3), 1), ((10, 48, 10), 1), ((10, 52, 10), 2), ((11, 64, 13), 2)])
def test_product(shape, passes, monkeypatch):
    s = _solver(shape, False)
    u = torch.from_numpy(np.random.default_rng(2).standard_normal(s.numDOFs)).cuda()
    for fp32 in (False, True):
        monkeypatch.delenv("TOPGPU_COARSE_TWOPASS_MIN", raising=False)
        n, y = _launches(s, lambda: s.matvec(0, u, fp32=fp32))
        assert n == 1 + passes + fp32          # onto the grid, the product; in single back from the grid
        other = "0" if passes == 1 else "1000000"
        monkeypatch.setenv("TOPGPU_COARSE_TWOPASS_MIN", other)
        q = _solver(shape, False)
        k, z = _launches(q, lambda: q.matvec(0, u, fp32=fp32))
        assert k == n + (1 if passes == 1 else -1) and torch.equal(y, z)


@pytest.mark.parametrize("mixed", [False, True])
def test_batch(mixed):
    """Three load cases on a model of 272 CTAs: one wave a right-hand side (the form
    in double), more than one over all three (single); every solve as by itself."""
    s = _solver((10, 20, 13), mixed, 3)
    U, its, _ = s.pcg_all()
    n = s.numDOFs
    F = s.mesh.get(0, "F").reshape(3, n)
    for k in range(3):
        Uk, ik, rk = s.pcg(k)
        assert rk < 1e-8
        b = torch.from_numpy(F[k]).cuda()
        # both solve to 1e-8 of the right-hand side, in single with sums grouped another way
        for x in (Uk, U[k * n:(k + 1) * n]):
            assert float((b - s.matvec(0, x)).norm()) < 2e-8 * float(b.norm())
        if not mixed:
            assert ik == its[k] and torch.equal(U[k * n:(k + 1) * n], Uk)
