"""Super-element kernels at the edges of their work splits: the density
filter's eight- and four-row threads with ragged last rows and every remainder
of its four-tap groups, element matrices of a count that is no multiple of
a CTA's, and the level-0 product's two passes against its one-pass kernel."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _to_fine(v, ny, nx, nz):
    f = np.zeros((4 * ny, 4 * nx, 4 * nz))
    for q in range(64):
        f[q % 4::4, q // 4 % 4::4, q // 16::4] = v[q::64].reshape((ny, nx, nz), order="F")
    return f


def _solver(shape, mixed=False):
    from top_gpu_on_matlab_b200.fea import Mesh, Solver
    m = Mesh(np.ones(shape, bool), control=20000, super_element=1)
    m.apply_optcase(1)
    return Solver(m, E0=1.0, Emin=1e-9, penal=3.0, tol=1e-8, maxIT=800, omega=0.6, mixed=mixed)


# taps 2R + 1 = 3, 7, 13, 5: R = ceil(4 rMin) - 1
@pytest.mark.parametrize("shape,rmin", [((3, 5, 3), 0.4), ((5, 7, 4), 1.0), ((11, 40, 12), np.sqrt(3)), ((13, 40, 12), 0.7)])
@pytest.mark.parametrize("mode", [0, 1])
def test_density_filter_shapes(shape, rmin, mode):
    from scipy import ndimage
    ny, nx, nz = shape
    s = _solver(shape)
    s.super_filter_setup(2.0)                   # a later setup replaces an earlier one
    s.super_filter_setup(rmin)
    v = np.random.default_rng(mode).random(64 * ny * nx * nz)
    out = s.super_filter(torch.from_numpy(v).cuda(), mode).cpu().numpy()
    r = 4 * rmin
    d = np.arange(1 - int(np.ceil(r)), int(np.ceil(r)))
    DY, DX, DZ = np.meshgrid(d, d, d, indexing="ij")
    h = np.maximum(0, r - np.sqrt(DY ** 2 + DX ** 2 + DZ ** 2))
    Hs = ndimage.correlate(np.ones((4 * ny, 4 * nx, 4 * nz)), h, mode="constant")
    g = _to_fine(v, ny, nx, nz)
    ref = ndimage.correlate(g / Hs, h, mode="constant") if mode == 0 else ndimage.correlate(g, h, mode="constant") / Hs
    assert np.abs(_to_fine(out, ny, nx, nz) - ref).max() <= 1e-12 * np.abs(ref).max()


def test_element_matrices_of_a_ragged_count():
    shape = (3, 5, 3)                           # 45 elements, 9 of them with fixed DOFs
    o = O.Model(np.ones(shape, bool), control=20000, super_element=1)
    o.apply_optcase(1)
    o.set_material(1.0, 1e-9, 3.0)
    s = _solver(shape)
    x = 0.1 + 0.9 * np.random.default_rng(5).random(64 * 45)
    o.set_density(x)
    o.assemble()
    s.set_density(torch.from_numpy(x).cuda())
    s.assemble()
    K, ref = s.Ks(0).cpu().numpy().reshape(576, -1, order="F"), o.K_mat()
    free = o.mapUniqueKes() == 0
    assert np.abs(K[:, free] - ref[:, free]).max() < 1e-13 * np.abs(ref).max()
    u = np.random.default_rng(6).standard_normal(o.level(0).numDOFs)     # the others through the product
    y, yo = s.matvec(0, torch.from_numpy(u).cuda()).cpu().numpy(), o.matvec(0, u)
    assert np.abs(y - yo).max() < 1e-12 * np.abs(yo).max()


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("shape", [(3, 5, 3), (10, 33, 7)])
def test_two_pass_level0_product_changes_no_result(shape, mixed, monkeypatch):
    x = torch.from_numpy(0.1 + 0.9 * np.random.default_rng(7).random(64 * int(np.prod(shape)))).cuda()
    outs = []
    for twoPassMin in ("0", "1000000"):
        monkeypatch.setenv("TOPGPU_COARSE_TWOPASS_MIN", twoPassMin)
        s = _solver(shape, mixed)
        s.set_density(x)
        s.assemble()
        u = torch.from_numpy(np.random.default_rng(8).standard_normal(s.numDOFs)).cuda()
        outs.append([s.matvec(0, u), s.matvec(0, u, fp32=True), s.vcycle(u)])
    for a, b in zip(*outs):
        assert torch.equal(a, b)
