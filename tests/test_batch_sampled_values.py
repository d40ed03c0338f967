"""Sampled batches of blocks return the same Ritz values whatever is changed in the kernel's layout or
the run's tiling: batches in which some blocks are singular to FP32, so that another order of sums gives
other values (tests/golden/sampled_batches.py), against the values on record.

Tolerance: 1e-6 of a matrix's λ (a block that is not singular moves by FP32 rounding, 1e-7, at most;
one that is moves by 1e-3 and more).
"""
from pathlib import Path

import numpy as np
import pytest

from golden.sampled_batches import BATCHES, run

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).parent / "golden" / "sampled_batches.npz"


@pytest.mark.parametrize("name", sorted(BATCHES))
def test_ritz_values_on_record(amm_lib, name):
    with np.load(GOLDEN) as g:
        lam, iters = g[name + "_lam"], g[name + "_iters"]
    got, got_iters = run(name)
    assert np.array_equal(got_iters, iters)
    ok = iters > 0
    assert np.array_equal(np.isnan(got), np.isnan(lam)) and ok.sum() > 0.8 * len(ok)
    off = np.abs(got[ok] - lam[ok]) / lam[ok][:, :1]
    assert off.max() < 1e-6, (int(np.argmax(off.max(1))), float(off.max()))


def test_wide_plan_that_the_caller_asked_for(amm_lib):
    """wide = 1 plans the wide launch by work alone, also over matrices of few picks."""
    import torch
    from eigenvaluecomputation_by_amm_b200 import BatchSolver
    g = torch.Generator(device="cuda").manual_seed(1)
    mats = [torch.randn(n, 512, device="cuda", generator=g).t() for n in [400] * 2 + [64] * 400]
    for c_divisor in (0, 8):
        solver = BatchSolver(mats, nvec=8, max_iter=8, tol=0.0, c_divisor=c_divisor,
                             vr_period=4 if c_divisor else 0, tile_gc=4, cluster=1, wide=1)
        solver.run()
        torch.cuda.synchronize()
        assert solver.wide_plan()["count"] == 2
        solver.close()
