"""Exact batches of 4 vectors are multiplied through A in FP32 whatever tiling the library takes: the
same bits as with that tile shape fixed, one launch a run, and no memory for C = A·Aᵀ (whose products are
less accurate than FP32 ones: λ's rms error 7.8e-8 against 6.6e-8)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_products_read_a(amm_lib):
    from eigenvaluecomputation_by_amm_b200 import BatchSolver
    g = torch.Generator(device="cuda").manual_seed(2)
    mats = [torch.randn(n, m, device="cuda", generator=g).t()
            for m, n in [(64, 900), (128, 2000), (260, 1000), (512, 2560)]]
    kw = dict(nvec=4, max_iter=20, tol=0.0, cluster=1, wide=-1)
    a = BatchSolver(mats, **kw)
    a.run()
    before = amm_lib.amm_kernel_launch_count()
    a.run()
    torch.cuda.synchronize()
    assert amm_lib.amm_kernel_launch_count() - before == 1
    b = BatchSolver(mats, tile_gc=a.tile_choice()[1], **kw)
    b.run()
    assert torch.equal(a.lam, b.lam) and torch.equal(a.vectors, b.vectors)
    a.close()
    b.close()
