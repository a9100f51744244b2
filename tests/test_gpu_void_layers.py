"""Models that leave whole layers, tiles or vector chunks void: the level-0
product's layer ranges and the PCG vector kernels' chunk lists skip them.  The
product against the staged kind, which visits every layer (FP64: the same
operations in the same order), and PCG, single and batched, against the
launches of a solver on the same model cut out of a larger padded box."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _mask(name):
    if name == "slab":              # z layers 0-4 and 13-19 void, the padding besides
        m = np.zeros((18, 40, 20), bool)
        m[:, :, 5:13] = True
    elif name == "corner":          # one tile column of many solid: most tiles void at every layer
        m = np.zeros((40, 70, 24), bool)
        m[:9, :, :6] = True
    elif name == "two":             # two separate z ranges joined by a bar
        m = np.zeros((20, 36, 40), bool)
        m[:, :, :6] = m[:, :, 30:37] = True
        m[4:10, 5:12, :37] = True
    else:                           # ragged box: void only in the padding
        m = np.ones((9, 33, 17), bool)
    return m


def _bc(m, mesh, loads):
    lv = mesh.info()[0]
    NY, NX = lv["resY"] + 1, lv["resX"] + 1
    fwd = mesh.get(0, "nodMapForward")
    act = np.flatnonzero(fwd)
    X = (act // NY) % NX
    fix = np.column_stack([fwd[act[X == 0]], np.ones((int((X == 0).sum()), 3))]).astype(float)
    end = fwd[act[X == X.max()]]
    r = np.random.default_rng(3)
    return fix, [np.column_stack([end, r.standard_normal((len(end), 3)) / len(end)]) for _ in range(loads)]


def _solver(name, mixed, loads=1):
    from top_gpu_on_matlab_b200.fea import Mesh, Solver
    m = _mask(name)
    mesh = Mesh(m, control=400)
    fix, ld = _bc(m, mesh, loads)
    mesh.apply_bc(fix, ld)
    s = Solver(mesh, E0=1.0, Emin=1e-9, penal=3.0, tol=1e-8, maxIT=800, omega=0.6, mixed=mixed)
    x = 0.4 + 0.6 * np.random.default_rng(4).random(s.num_design)
    s.set_density(torch.from_numpy(x).cuda())
    s.assemble()
    return s, m, x, fix, ld


@pytest.mark.parametrize("name", ["slab", "corner", "two", "ragged"])
def test_product_skips_void_layers(name):
    s, m, x, fix, ld = _solver(name, False)
    u = torch.from_numpy(np.random.default_rng(5).standard_normal(s.numDOFs)).cuda()
    out = []
    for kind, ty, tx in ((3, 16, 8), (3, 16, 16), (1, 16, 8)):
        s.set_l0_kernel(False, kind, ty, tx, 12 * 148)
        out.append(s.matvec(0, u))
    assert torch.equal(out[0], out[2]) and torch.equal(out[1], out[2])
    o = O.Model(m, control=400)
    o.apply_bc(fix, ld)
    o.set_material(1.0, 1e-9, 3.0)
    o.set_density(x)
    ref = o.matvec(0, u.cpu().numpy())
    assert np.abs(out[0].cpu().numpy() - ref).max() < 1e-13 * np.abs(ref).max()


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("name", ["slab", "corner", "two", "ragged"])
def test_pcg_with_void_chunks(name, mixed):
    """The solution solves the system (residual through the product that visits
    every layer), and a batch of five load cases equals its single solves."""
    s, m, x, fix, ld = _solver(name, mixed, loads=5)
    U, its, res = s.pcg_all()
    n = s.numDOFs
    F = s.mesh.get(0, "F").reshape(5, n)
    for k in range(5):
        Uk, ik, rk = s.pcg(k)
        assert ik == its[k] and torch.equal(U[k * n:(k + 1) * n], Uk)
    s.set_l0_kernel(False, 1, 16, 8, 12 * 148)
    for k in range(5):
        b = torch.from_numpy(F[k]).cuda()
        r = b - s.matvec(0, U[k * n:(k + 1) * n])
        # the solve's own (recurrence's) residual, converged or at the iteration
        # limit; the true one follows it to rounding
        assert float(r.norm()) < 2 * res[k] * float(b.norm())


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("name", ["slab", "corner", "two"])
def test_same_model_in_a_larger_box(name, mixed):
    """The model with 17 more void layers around it in z (the node order is the
    same): equal products, V-cycles to rounding, and each solver's solution
    solves the other's system."""
    from top_gpu_on_matlab_b200.fea import Mesh, Solver
    m = _mask(name)
    sol = []
    for extra in (0, 17):
        mk = np.concatenate([m, np.zeros(m.shape[:2] + (extra,), bool)], 2)
        mesh = Mesh(mk, control=400)
        fix, ld = _bc(m, mesh, 1)
        mesh.apply_bc(fix, ld)
        s = Solver(mesh, E0=1.0, Emin=1e-9, penal=3.0, tol=1e-9, maxIT=800, omega=0.4, mixed=mixed)
        s.set_density(torch.from_numpy(0.4 + 0.6 * np.random.default_rng(4).random(s.num_design)).cuda())
        s.assemble()
        u = torch.from_numpy(np.random.default_rng(5).standard_normal(s.numDOFs)).cuda()
        U, _, res = s.pcg(0)
        assert res < 1e-9
        sol.append((s, s.matvec(0, u), s.vcycle(u), U))
    (s0, y0, z0, U0), (s1, y1, z1, U1) = sol
    assert torch.equal(y0, y1)
    assert float((z0 - z1).abs().max()) < (1e-5 if mixed else 1e-11) * float(z0.abs().max())
    b = torch.from_numpy(s0.mesh.get(0, "F")).cuda()
    for s, U in ((s0, U1), (s1, U0)):
        assert float((b - s.matvec(0, U)).norm()) < 2e-9 * float(b.norm())
