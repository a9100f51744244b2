"""The grid size from which void layers and vector chunks are left out: below it,
above it and with the line moved past the model the solver gives the same
products and V-cycles, and solves that agree (a solve's dot products add the
same values, in another grouping)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _solver(shape, solid, mixed):
    from top_gpu_on_matlab_b200.fea import Mesh, Solver
    mask = np.zeros(shape, bool)
    mask[solid] = True
    mesh = Mesh(mask, control=400)
    lv = mesh.info()[0]
    NY, NX = lv["resY"] + 1, lv["resX"] + 1
    fwd = mesh.get(0, "nodMapForward")
    act = np.flatnonzero(fwd)
    X = act // NY % NX
    fix, end = fwd[act[X == X.min()]], fwd[act[X == X.max()]]
    r = np.random.default_rng(1)
    mesh.apply_bc(np.column_stack([fix, np.ones((len(fix), 3))]).astype(float),
                  [np.column_stack([end, r.standard_normal((len(end), 3)) / len(end)])])
    s = Solver(mesh, E0=1.0, Emin=1e-9, penal=3.0, tol=1e-10, maxIT=800, omega=0.4, mixed=mixed)
    s.set_density(torch.from_numpy(0.4 + 0.6 * r.random(s.num_design)).cuda())
    s.assemble()
    return s


SLAB = np.s_[:, :, 5:13]
# level-0 slots: 33 thousand (below 48 x 1024), 109 thousand, a ragged box of 57 thousand
@pytest.mark.parametrize("shape,solid", [((18, 40, 20), SLAB), ((36, 40, 60), np.s_[:30, 3:, 7:40]), ((17, 65, 18), np.s_[:, :, :])])
@pytest.mark.parametrize("mixed", [False, True])
def test_void_line(shape, solid, mixed, monkeypatch):
    out, sol = [], []
    for line in (None, "0", "1000000000"):
        if line is None:
            monkeypatch.delenv("TOPGPU_VOID_MIN_SLOTS", raising=False)
        else:
            monkeypatch.setenv("TOPGPU_VOID_MIN_SLOTS", line)
        s = _solver(shape, solid, mixed)
        u = torch.from_numpy(np.random.default_rng(2).standard_normal(s.numDOFs)).cuda()
        out.append([s.matvec(0, u), s.matvec(0, u, fp32=True), s.vcycle(u)])
        sol.append(s.pcg(0))
    for o in out[1:]:
        for a, b in zip(o, out[0]):
            assert torch.equal(a, b)
    # each solution's own residual through one product, and the line's default equal to one of the two forms
    F = torch.from_numpy(s.mesh.get(0, "F")).cuda()
    for U, its, res in sol:
        assert float((F - s.matvec(0, U)).norm()) < 2 * max(res, 1e-10) * float(F.norm())
    assert any(torch.equal(sol[0][0], sol[k][0]) for k in (1, 2))
