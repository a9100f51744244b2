"""The scatter gateway where neighbouring lanes hold the same node: a box's own
numbering, random ids with many repeats, one node for all, and ids out of range, at
sizes around a warp and a CTA.  Whole-numbered values: every sum is exact, so the
result equals numpy's to the last bit in any order."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("ids", ["random", "few", "one", "line", "out"])
def test_scatter_counts_every_value_once(ids, dt):
    from top_gpu_on_matlab_b200 import mex
    r = np.random.default_rng(5)
    for ne in (1, 2, 31, 32, 33, 255, 257, 1000):
        nn = 2 * (ne + 1) * 4
        if ids == "line":                # a column of elements: the upper face is the next one's lower
            lower = 1 + np.arange(ne)[:, None] + (ne + 1) * np.arange(4)[None, :]
            eN = np.empty((ne, 8), np.int64)
            eN[:, [3, 2, 7, 6]], eN[:, [0, 1, 4, 5]] = lower, lower + 1
        else:
            top = {"random": nn, "few": 3, "one": 1, "out": nn}[ids]
            eN = r.integers(1, top + 1, (ne, 8))
        if ids == "out":
            eN[r.random((ne, 8)) < 0.3] = 0
            eN[r.random((ne, 8)) < 0.3] = nn + 1
        v = r.integers(-8, 9, (ne, 24)).astype(dt)
        Y0 = r.integers(-8, 9, (nn, 3)).astype(dt)
        ref = Y0.copy()
        for j in range(8):
            ok = (eN[:, j] >= 1) & (eN[:, j] <= nn)
            np.add.at(ref, eN[ok, j] - 1, v[ok, 3 * j:3 * j + 3])
        Y = mex.gpu_array(Y0)
        mex.Scattering_inplace(Y, mex.gpu_array(eN.astype(np.int32)), mex.gpu_array(v))
        assert np.array_equal(Y.cpu().numpy(), ref), (ids, ne)
