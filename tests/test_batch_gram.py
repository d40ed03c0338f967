"""Block products as C·X with C = A·Aᵀ formed on the tensor cores (amm_gram.cu), on the B200: sizes at
the edges of its 128 x 256 tiles, 32-column chunks and 4-row groups, against FP64 and against the
same batch with a fixed tile shape (products through A); rows past m holding NaN; a rebind; one launch
per matrix; sampled products with variance reduction, whose exact products take the same route.

Tolerances: λ within 1e-6 relative of FP64 (FP32 sums of 3-way BF16 products: 1e-7 measured, the
products through A 1.4e-7), Ritz values of the two routes within 2e-6 of λ.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# (m, n): one row group, one tile and one more row, two and three row blocks (the last tile of an odd
# one spans the diagonal), column remainders of a chunk, the largest m; n < m stays on A
SIZES = [(8, 300), (64, 33), (127, 256), (128, 257), (129, 500), (256, 700), (260, 1000),
         (385, 1203), (512, 640), (771, 1500), (2048, 2100), (500, 90)]


def _mats(sizes, seed, nan_rows=True):
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = []
    for m, n in sizes:
        ld = (m + 3) // 4 * 4 + 4
        buf = torch.full((n, ld), float("nan") if nan_rows else 0.0, device="cuda")
        buf[:, :m] = torch.randn(n, m, device="cuda", generator=g) * torch.exp(
            torch.randn(n, 1, device="cuda", generator=g))
        out.append(buf.t()[:m])
    return out




@pytest.mark.parametrize("nvec", [4, 8])
@pytest.mark.parametrize("cluster", [1, 4])
def test_products_by_c_match_products_through_a(amm_lib, nvec, cluster):
    from eigenvaluecomputation_by_amm_b200 import BatchSolver
    sizes = [s for s in SIZES if s[0] >= nvec]
    mats = _mats(sizes, seed=3)
    a = BatchSolver(mats, nvec=nvec, max_iter=24, tol=0.0, cluster=cluster)
    b = BatchSolver(mats, nvec=nvec, max_iter=24, tol=0.0, cluster=cluster, tile_gc=2)
    a.run()
    b.run()
    torch.cuda.synchronize()
    assert torch.equal(a.iters, b.iters)
    scale = b.lam[:, :1]
    assert float(((a.lam - b.lam).abs() / scale).max()) < 2e-6
    lam1, vec1 = a.lam.clone(), a.vectors.clone()
    a.run(each=True)                      # one launch per matrix: the same bits
    assert torch.equal(a.lam, lam1) and torch.equal(a.vectors, vec1)
    a.run()                               # and from the captured graph
    assert torch.equal(a.lam, lam1) and torch.equal(a.vectors, vec1)
    a.close()
    b.close()


def test_converged_lambda_vs_fp64_and_rebind(amm_lib):
    from eigenvaluecomputation_by_amm_b200 import BatchSolver
    first, second = _mats(SIZES, seed=5), _mats(SIZES, seed=6)
    bs = BatchSolver(first, nvec=8, max_iter=2000, tol=1e-6)
    for mats in (first, second):
        bs.set_matrices(mats)
        lam, _, iters = bs.run()
        torch.cuda.synchronize()
        assert int(iters.min()) > 0 and int(iters.max()) < 2000
        for i, A in enumerate(mats):
            A = A.double()
            w = torch.linalg.eigvalsh(A @ A.t())[-1]
            assert abs(float(lam[i] - w)) < 1e-6 * float(w), (SIZES[i], float(lam[i]), float(w))
    bs.close()


@pytest.mark.parametrize("cluster", [1, 2])
def test_variance_reduced_products_by_c(amm_lib, cluster):
    from eigenvaluecomputation_by_amm_b200 import BatchSolver
    sizes = [(64, 512), (130, 700), (300, 2048), (600, 4000)]
    mats = _mats(sizes, seed=9, nan_rows=False)
    kw = dict(nvec=8, max_iter=12, tol=0.0, c_divisor=4, vr_period=3, cluster=cluster)
    a, b = BatchSolver(mats, **kw), BatchSolver(mats, tile_gc=2, **kw)
    a.run()
    b.run()
    torch.cuda.synchronize()
    # the same picks (they depend on the seeds and the norms alone), so the same estimates
    assert float(((a.lam[:, 0] - b.lam[:, 0]).abs() / b.lam[:, 0]).max()) < 2e-6
    a.close()
    b.close()


def test_without_room_for_c_the_products_read_a():
    """C of all the matrices (206 GB) does not fit the device: the solver is made without it."""
    from eigenvaluecomputation_by_amm_b200 import BatchSolver
    A = torch.zeros(4096, 2048, device="cuda").t()
    free0 = torch.cuda.mem_get_info()[0]
    solver = BatchSolver([A] * 12288, nvec=8, max_iter=20, tol=0.0)
    assert free0 - torch.cuda.mem_get_info()[0] < 4 << 30
    solver.close()
