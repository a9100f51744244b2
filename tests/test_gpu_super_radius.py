"""The super-element density filter with radii up to several times the grid:
against the correlation with all its taps, and without the work and memory of the
taps that no two voxels of the grid are apart by."""
import numpy as np
import pytest
import torch

from tests.test_gpu_super_shapes import _solver, _to_fine

pytestmark = pytest.mark.gpu


# reach R = ceil(4 rMin) - 1 below, at and beyond the fine grid's extents (12, 20, 16)
@pytest.mark.parametrize("rmin", [2.6, 2.9, 3.1, 4.0, 5.0, 5.3])
@pytest.mark.parametrize("mode", [0, 1])
def test_radius_of_the_grids_size(rmin, mode):
    from scipy import ndimage
    ny, nx, nz = 3, 5, 4
    s = _solver((ny, nx, nz))
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
    # at most 3840 positive terms a sum, two sums and a division: 4e3 eps = 1e-12
    assert np.abs(_to_fine(out, ny, nx, nz) - ref).max() <= 1e-12 * np.abs(ref).max()


def test_taps_beyond_the_grid_cost_nothing():
    """24x64x24 fine grid, R = 47 and 79 (both past its extents in y and z): about the
    same taps meet the grid, so the time does not follow the radius's cube (4.7
    times) and the taps and the operand stay within a few times the grid."""
    s = _solver((6, 16, 6))
    v = torch.rand(s.num_design, dtype=torch.float64, device="cuda")
    ms = {}
    for rmin in (12.0, 20.0):
        free = torch.cuda.mem_get_info()[0]
        s.super_filter_setup(rmin)
        assert free - torch.cuda.mem_get_info()[0] < 32 << 20
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        times = []
        for _ in range(5):
            a.record()
            s.super_filter(v, 1)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        ms[rmin] = min(times)
    assert ms[20.0] < 3 * ms[12.0], ms
