"""The level-2 Galerkin gateway's two forms of Q = P' K0 P (from scratch memory
for one row block of cells or the allocation-free entry point, formed by each CTA
beyond that) give the same matrices bit for bit, both as the oracle's, over
row-block remainders, 64 and 8 children, with and without fixed DOFs (whose
cells are found by probing all of them); and the single-precision class, in
FP64 inside, within its storage rounding."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.test_zzzz_no_alloc import _col, _pch

pytestmark = pytest.mark.gpu


def _call(name, upMap, E, K0, P, mu, fr, fx, single=False):
    from top_gpu_on_matlab_b200._lib import TOP_F32, TOP_F64, check, lib
    dt = torch.float32 if single else torch.float64
    nE, nCh = upMap.shape
    nU = 0 if fr is None else fr.shape[1]
    t = [_col(upMap, torch.int32), _col(E, dt), _col(K0, dt), _col(P, dt), _col(mu, torch.int32)]
    u = [_col(a, dt) for a in (fr, fx)] if nU else []
    Ks = torch.full((576 * nE,), float("nan"), dtype=dt, device="cuda")
    check(getattr(lib(), name)(Ks.data_ptr(), *[a.data_ptr() for a in t], *([a.data_ptr() for a in u] if nU else [None, None]),
                               nE, nCh, E.size, nU, TOP_F32 if single else TOP_F64, None), name)
    return Ks.cpu().numpy().astype(np.float64)


# coarse cells 64 (one row block), 65 ..., 480: (ny / 4)(nx / 4)(nz / 4)
@pytest.mark.parametrize("shape", [(16, 16, 16), (20, 52, 4 * 4), (24, 40, 32)])
@pytest.mark.parametrize("fixed", [True, False])
def test_level2_paths(shape, fixed):
    m = O.Model(np.ones(shape, bool), control=20000)
    m.apply_optcase(1)
    L0, L1, L2 = m.level(0), m.level(1), m.level(2)
    E = 0.05 + np.random.default_rng(31).random(L0.numElements)
    fr, fx = m.uniqueKes() if fixed else (None, None)
    mu = m.mapUniqueKes() if fixed else np.zeros(L0.numElements, np.int32)
    args = (L1.elementUpwardMap, E, L0.Ke, _pch(4), mu, fr, fx)
    a, b = _call("top_assemble_ks_level2", *args), _call("top_assemble_ks_level2_noalloc", *args)
    assert np.array_equal(a, b)
    ref = O.assemble_ks_level2(*args).ravel(order="F")
    assert np.abs(a - ref).max() < 1e-13 * np.abs(ref).max()
    # single: inputs and result rounded to 24 bits (2^-24 each, products of three inputs), sums in FP64
    f = _call("top_assemble_ks_level2", *args, single=True)
    assert np.abs(f - ref).max() < 8 * 2.0 ** -24 * np.abs(ref).max()
    # eight children: GEMM rows 8..63 multiply zeros
    E2 = 0.2 + np.random.default_rng(32).random(L1.numElements)
    args2 = (L2.elementUpwardMap, E2, L1.Ke, _pch(2), np.zeros(L1.numElements, np.int32), None, None)
    a2, b2 = _call("top_assemble_ks_level2", *args2), _call("top_assemble_ks_level2_noalloc", *args2)
    assert np.array_equal(a2, b2) and np.isfinite(a2).all()


@pytest.mark.parametrize("single", [False, True])
def test_higher_level_with_void_children(single):
    """Cells whose first, last or every second child is void, a count that is no
    multiple of a CTA's four: the child prefetch skips them."""
    from top_gpu_on_matlab_b200 import mex
    dt = np.float32 if single else np.float64
    rng = np.random.default_rng(33)
    nf, nc = 37, 11
    A = rng.standard_normal((24, 24, nf))
    Kp = np.einsum("ijk,ljk->ilk", A, A)
    up = rng.integers(1, nf + 1, (nc, 8)).astype(np.int32)
    up[0, 0] = up[1, 7] = 0
    up[2, ::2] = 0
    up[3, :] = 0
    ref = O.assemble_ks_higher(up, Kp, _pch(2))
    Ks = mex.zeros((24, 24, nc), dtype=torch.float32 if single else torch.float64)
    mex.assembleKs_higherLevel_inplace(Ks, mex.gpu_array(up), mex.gpu_array(Kp.astype(dt)), mex.gpu_array(_pch(2).astype(dt)))
    tol = 8 * 2.0 ** -24 if single else 1e-13
    assert np.abs(mex.gather(Ks).astype(np.float64) - ref).max() < tol * np.abs(ref).max()
