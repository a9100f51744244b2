"""A call that ends with a non-finite scalar (TOP_ERR_NAN) leaves nothing behind:
the next call on the same solver gives what a solver that never failed gives,
bit for bit.  Models with void layers, padding and guard slots, whose vectors
are zero there and are not written by every kernel."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

BAD = [float("nan"), float("inf"), 1e200]      # 1e200: finite, its square is not


@pytest.fixture(autouse=True)
def _void_left_out(monkeypatch):
    monkeypatch.setenv("TOPGPU_VOID_MIN_SLOTS", "0")       # the models are small


def _mesh(loads=1):
    from top_gpu_on_matlab_b200.fea import Mesh
    mask = np.zeros((18, 40, 20), bool)
    mask[:, :, 5:13] = True
    m = Mesh(mask, control=400)
    lv = m.info()[0]
    NY, NX = lv["resY"] + 1, lv["resX"] + 1
    fwd = m.get(0, "nodMapForward")
    act = np.flatnonzero(fwd)
    X = act // NY % NX
    fix, end = fwd[act[X == 0]], fwd[act[X == X.max()]]
    r = np.random.default_rng(1)
    m.apply_bc(np.column_stack([fix, np.ones((len(fix), 3))]).astype(float),
               [np.column_stack([end, r.standard_normal((len(end), 3)) / len(end)]) for _ in range(loads)])
    return m


def _solver(m, mixed, assemble=True):
    from top_gpu_on_matlab_b200.fea import Solver
    s = Solver(m, E0=1.0, Emin=1e-9, penal=3.0, tol=1e-8, maxIT=400, omega=0.6, mixed=mixed)
    if assemble:
        s.set_density(_density(s))
        s.assemble()
    return s


def _density(s):
    return torch.from_numpy(0.4 + 0.6 * np.random.default_rng(2).random(s.num_design)).cuda()


def _fails(call):
    from top_gpu_on_matlab_b200._lib import TOP_ERR_NAN, TopGpuError
    with pytest.raises(TopGpuError) as e:
        call()
    assert e.value.status == TOP_ERR_NAN


@pytest.mark.parametrize("bad", BAD)
def test_filter(bad):
    m = _mesh()
    fresh, s = _solver(m, False, False), _solver(m, False, False)
    for q in (fresh, s):
        q.filter_setup(2.5)
    x = _density(s)
    ref, its = fresh.filter(x)
    y = x.clone()
    y[7] = bad
    for _ in range(2):
        _fails(lambda: s.filter(y))
        out, k = s.filter(x)
        assert k == its and torch.equal(out, ref)


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("bad", BAD[:2])
def test_pcg_right_hand_side(mixed, bad):
    m = _mesh()
    fresh, s = _solver(m, mixed), _solver(m, mixed)
    U0, its0, _ = fresh.pcg(0)
    b = torch.zeros(s.numDOFs, dtype=torch.float64, device="cuda")
    b[5 * 3 + 1] = bad
    for _ in range(2):
        _fails(lambda: s.pcg(b=b))
        U, its, _ = s.pcg(0)
        assert its == its0 and torch.equal(U, U0)


@pytest.mark.parametrize("mixed", [False, True])
def test_batched_pcg_warm_start(mixed):
    """one of three load cases starts from a vector with a NaN"""
    from top_gpu_on_matlab_b200._lib import TopGpuError
    m = _mesh(3)
    fresh, s = _solver(m, mixed), _solver(m, mixed)
    U0, its0, _ = fresh.pcg_all()
    W = torch.zeros_like(U0)
    W[s.numDOFs + 11] = float("nan")
    with pytest.raises(TopGpuError):
        s.pcg_all(W)
    U, its, _ = s.pcg_all()
    assert its == its0 and torch.equal(U, U0)


@pytest.mark.parametrize("mixed", [False, True])
def test_density(mixed):
    m = _mesh()
    fresh, s = _solver(m, mixed), _solver(m, mixed)
    x = _density(s)
    y = x.clone()
    y[7] = float("nan")
    s.set_density(y)
    _fails(s.assemble)
    s.set_density(x)
    s.assemble()
    U0, its0, _ = fresh.pcg(0)
    U, its, _ = s.pcg(0)
    assert its == its0 and torch.equal(U, U0)


@pytest.mark.parametrize("mixed", [False, True])
def test_operators(mixed):
    """The V-cycle and the product on a vector with a NaN, through the level-0
    kernel that visits every layer; then through the one that leaves the void
    layers out."""
    m = _mesh()
    out = []
    for bad in (0.0, float("nan")):
        s = _solver(m, mixed)
        s.set_l0_kernel(False, 1, 16, 8, 12 * 148)
        s.set_l0_kernel(True, 1, 16, 8, 12 * 148)
        u = torch.from_numpy(np.random.default_rng(3).standard_normal(s.numDOFs)).cuda()
        v = u.clone()
        if bad != 0.0:
            v[:] = bad
        s.matvec(0, v), s.matvec(0, v, fp32=True), s.vcycle(v)
        s.set_l0_kernel(False, 3, 16, 8, 12 * 148)
        s.set_l0_kernel(True, 3, 16, 8, 12 * 148)
        out.append([s.matvec(0, u), s.matvec(0, u, fp32=True), s.vcycle(u), s.pcg(0)[0]])
    for a, b in zip(*out):
        assert torch.equal(a, b)


def test_single_product_before_a_double_vcycle():
    """y = K u in single through a kernel that visits every layer, on a vector with
    a NaN; then the FP64 V-cycle, whose kernel leaves the void layers out."""
    m = _mesh()
    out = []
    for bad in (0.0, float("nan")):
        s = _solver(m, False)
        s.set_l0_kernel(True, 1, 16, 8, 12 * 148)
        s.set_l0_kernel(False, 3, 16, 8, 12 * 148)
        u = torch.from_numpy(np.random.default_rng(3).standard_normal(s.numDOFs)).cuda()
        s.matvec(0, torch.full_like(u, bad), fp32=True)
        out.append(s.vcycle(u))
    assert torch.equal(*out)
