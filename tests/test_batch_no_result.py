"""The vector of a matrix without a result (here: the zero matrix) is zeros after the first run, whatever
the memory held before; the matrices beside it have theirs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [{}, dict(c_divisor=8, vr_period=4), dict(nvec=4)])
def test_vector_without_a_result(amm_lib, kw):
    from eigenvaluecomputation_by_amm_b200 import BatchSolver
    g = torch.Generator(device="cuda").manual_seed(6)
    good = torch.randn(700, 64, device="cuda", generator=g).t()
    zero = torch.zeros(700, 64, device="cuda").t()
    filler = [torch.ones(128, device="cuda") for _ in range(16)]
    del filler                            # the next allocations of this size find ones
    solver = BatchSolver([good, zero], max_iter=12, tol=0.0, **{"nvec": 8, **kw})
    solver.run()
    torch.cuda.synchronize()
    assert solver.iters.tolist() == [12, -1]
    assert bool(torch.isnan(solver.lam[1]).all()) and bool(torch.isfinite(solver.lam[0]).all())
    assert bool((solver.vector(1) == 0).all())
    assert abs(float(solver.vector(0).norm()) - 1) < 1e-5
    solver.close()
