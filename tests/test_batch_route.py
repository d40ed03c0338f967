"""Which products an exact batch of 8 vectors takes: through C = A·Aᵀ (one launch more a run, which
forms C) only where that is less work.

On a B200, 20 products of 148 or 296 equal matrices, time through C over time through A: 1024 x 614
1.26, 512 x 307 1.10, 2048 x 1229 1.41 (these must read A); 512 x 2560 0.35, 256 x 1280 0.42,
1024 x 5120 0.41 (these must go through C).  A block that converges in two products must read A at a size
where forming C takes as long as four products (the autotuner times both).
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _launches(lib, solver):
    solver.run()
    before = lib.amm_kernel_launch_count()
    solver.run()
    torch.cuda.synchronize()
    return lib.amm_kernel_launch_count() - before


@pytest.mark.parametrize("m,n,by_c", [(1024, 614, False), (512, 307, False), (2048, 1229, False),
                                      (2048, 512, False), (512, 2560, True), (256, 1280, True),
                                      (1024, 5120, True)])
def test_equal_matrices(amm_lib, m, n, by_c):
    from eigenvaluecomputation_by_amm_b200 import BatchSolver
    g = torch.Generator(device="cuda").manual_seed(m + n)
    A = torch.randn(n, m, device="cuda", generator=g).t()
    solver = BatchSolver([A] * (296 if m <= 512 else 148), nvec=8, max_iter=20, tol=0.0, wide=-1)
    assert _launches(amm_lib, solver) == (2 if by_c else 1)
    solver.close()


def test_few_products_to_a_tolerance(amm_lib):
    from eigenvaluecomputation_by_amm_b200 import BatchSolver
    g = torch.Generator(device="cuda").manual_seed(4)
    mats = []
    for _ in range(148):
        buf = 1e-3 * torch.randn(4096, 512, device="cuda", generator=g)
        buf[:8] *= 1e6 * torch.arange(8, 0, -1, device="cuda")[:, None]
        mats.append(buf.t())
    solver = BatchSolver(mats, nvec=8, max_iter=1000, tol=1e-6, wide=-1)
    assert _launches(amm_lib, solver) == 1
    assert 0 < int(solver.iters.min()) and int(solver.iters.max()) < 8
    A = mats[5].double()
    w = torch.linalg.eigvalsh(A @ A.t())[-1]
    assert abs(float(solver.lam[5, 0] - w)) < 1e-6 * float(w)
    solver.close()
