"""A tile copy of the packed coarsest product withheld by the test hook: its
bounded wait runs out (one second), the V-cycle reports TOP_ERR_CUDA, and the
next calls give what a solver that never failed gives, bit for bit."""
import time

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
def test_packed_product_wait_gives_up_and_reports(mixed, monkeypatch):
    from top_gpu_on_matlab_b200._lib import TOP_ERR_CUDA, TopGpuError
    from top_gpu_on_matlab_b200.fea import Mesh, Solver
    monkeypatch.setenv("TOPGPU_COARSE_TWOPASS_MIN", "1000000")     # the coarse levels' products take no tile copies
    m = Mesh(np.ones((56, 88, 56), bool), control=20000)
    assert 3 * m.info()[-1]["numNodes"] == 2304
    m.apply_optcase(1)
    x = torch.from_numpy(0.2 + 0.7 * np.random.default_rng(4).random(m.info()[0]["numElements"])).cuda()
    r = torch.from_numpy(np.random.default_rng(5).standard_normal(3 * m.info()[0]["numNodes"])).cuda()
    fresh, s = (Solver(m, E0=1.0, Emin=1e-9, penal=3.0, tol=1e-6, maxIT=400, omega=0.4, mixed=mixed) for _ in range(2))
    for q in (fresh, s):
        q.set_density(x)
        q.assemble()
    ref = fresh.vcycle(r)
    s.test_withhold_tile()
    t = time.perf_counter()
    with pytest.raises(TopGpuError) as e:
        s.vcycle(r)
    assert e.value.status == TOP_ERR_CUDA and "tile copy did not complete" in str(e.value)
    assert 0.9 < time.perf_counter() - t < 5
    assert torch.equal(s.vcycle(r), ref)
    U0, its0, _ = fresh.pcg(0)
    U1, its1, _ = s.pcg(0)
    assert its0 == its1 and torch.equal(U0, U1)
