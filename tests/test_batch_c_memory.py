"""C = A·Aᵀ of an exact batch takes a small part of the device's free memory: all of it where an eighth of
that holds it, else the matrices that save most, up to a 48th.  With 1.2 GiB free: 20 matrices of 1024 x
5120 (80 MiB of C) have all theirs, of 60 (240 MiB) some do, and both runs return the Ritz values of the
products through A within 2e-6 of λ (FP32 rounding, the tolerance of test_batch_gram)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
MIB = 1 << 20


def _free():
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_part_of_the_batch_has_room(amm_lib):
    from eigenvaluecomputation_by_amm_b200 import BatchSolver
    g = torch.Generator(device="cuda").manual_seed(8)
    mats = [torch.randn(5120, 1024, device="cuda", generator=g).t() for _ in range(2)]
    kw = dict(nvec=8, max_iter=60, tol=0.0, cluster=2, wide=-1)
    first = BatchSolver(mats, **kw)       # loads what is loaded at a first run
    first.run()
    first.close()
    want = {}
    for count in (20, 60):                # (a start block follows the matrix's place in the batch)
        by_a = BatchSolver([mats[i % 2] for i in range(count)], tile_gc=8, **kw)
        by_a.run()
        want[count] = by_a.lam.clone()
        by_a.close()
    filler = torch.empty(_free() - 1228 * MIB, dtype=torch.uint8, device="cuda")
    try:
        for count, lo, hi in ((20, 80, 100), (60, 12, 40)):
            batch = [mats[i % 2] for i in range(count)]
            before = _free()
            solver = BatchSolver(batch, **kw)
            assert lo * MIB <= before - _free() <= hi * MIB, (before - _free()) / MIB
            launches = amm_lib.amm_kernel_launch_count()
            solver.run()
            torch.cuda.synchronize()
            assert amm_lib.amm_kernel_launch_count() - launches == 2   # C is formed
            ref = want[count]
            assert float(((solver.lam - ref).abs() / ref[:, :1]).max()) < 2e-6
            solver.close()
    finally:
        del filler
        torch.cuda.empty_cache()
