"""The PDE filter's product at the edges of its 16 x 16 tiles (15 x 15 output
nodes) and z-segments, on full and partly void models, through the whole
filter: against a sparse direct solve of the same Helmholtz system (the
reference's element matrix, natural-coordinate gradients, unit weights)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CORNERS = [(1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 0), (1, 0, 1), (1, 1, 1), (0, 1, 1), (0, 0, 1)]


def _reference(mask, x, rmin):
    import scipy.sparse as sp
    from scipy.sparse.linalg import spsolve
    s = np.array([(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1)], float)
    K = np.zeros((8, 8))
    for p in np.ndindex(2, 2, 2):
        f = 1 + s * ((np.array(p) * 2 - 1) / np.sqrt(3.0))
        N = f.prod(1) / 8
        dN = np.stack([s[:, k] * np.delete(f, k, 1).prod(1) / 8 for k in range(3)])
        K += (rmin / 2 / np.sqrt(3.0)) ** 2 * dN.T @ dN + np.outer(N, N) / 8
    ny, nx, nz = mask.shape
    e = np.flatnonzero(mask.ravel(order="F"))
    ey, ex, ez = e % ny, e // ny % nx, e // (ny * nx)
    nod = np.stack([(ey + dy) + (ny + 1) * ((ex + dx) + (nx + 1) * (ez + dz)) for dy, dx, dz in CORNERS], 1)
    used, nod = np.unique(nod, return_inverse=True)
    nod = nod.reshape(-1, 8)
    n = len(used)
    A = sp.csc_matrix((np.tile(K.ravel(), len(e)), (np.repeat(nod, 8, 1).ravel(), np.tile(nod, (1, 8)).ravel())), shape=(n, n))
    b = np.bincount(nod.ravel(), np.repeat(x / 8, 8), n)
    return spsolve(A, b)[nod].mean(1)


@pytest.mark.parametrize("shape,void", [((3, 3, 3), False), ((14, 15, 16), False), ((15, 29, 5), False), ((30, 14, 31), False), ((16, 31, 9), True)])
def test_filter_at_tile_edges(shape, void):
    from top_gpu_on_matlab_b200.fea import Mesh, Solver
    mask = np.ones(shape, bool)
    if void:
        mask[5:9, 10:20, :] = False
        mask[:, 3, 4] = False
    m = Mesh(mask, control=20000)
    lv = m.info()[0]
    NY, NX = lv["resY"] + 1, lv["resX"] + 1
    fwd = m.get(0, "nodMapForward")
    act = np.flatnonzero(fwd)
    X = act // NY % NX
    m.apply_bc(np.column_stack([fwd[act[X == 0]], np.ones((int((X == 0).sum()), 3))]).astype(float),
               [np.array([[fwd[act[X == X.max()]][0], 0, 0, -1.0]])])
    s = Solver(m, E0=1.0, Emin=1e-9, penal=3.0, tol=1e-11, maxIT=800, omega=0.6)
    x = np.random.default_rng(1).random(int(mask.sum()))
    for rmin in (1.5, 3.0):
        s.filter_setup(rmin)
        out, its = s.filter(torch.from_numpy(x).cuda())
        ref = _reference(mask, x, rmin)
        # residual 1e-12 of the right-hand side on a system of condition below 1e3
        assert np.abs(out.cpu().numpy() - ref).max() < 1e-9 * np.abs(ref).max(), its
