"""Sampled batches whose blocks can be singular, and the results to keep (sampled_batches.npz).

Small matrices with a few picks per product: a product sampled before the first memo has the rank of
its distinct picks, and the vectors past that rank are rounding, so that the order of the sums shows
in the Ritz values that follow.  The file holds the Ritz values and iteration counts of commit
3a8de82 on a B200; to write it again, run this file in a built tree of that commit:

    python sampled_batches.py OUT.npz
"""
import math
import sys

import numpy as np

# name: (matrices, rows from, to, columns from, to, keyword arguments of the solver)
BATCHES = {
    "k8_vr": (111, 16, 120, 64, 700, dict(nvec=8, max_iter=9, c_divisor=8, vr_period=4)),
    "k8_vr_fixed": (60, 16, 120, 64, 700,
                    dict(nvec=8, max_iter=20, c_divisor=8, vr_period=4, tile_gc=2, cluster=2)),
    "k8_plain": (60, 16, 120, 64, 700, dict(nvec=8, max_iter=6, c_divisor=8, cluster=1)),
    "k4_vr": (80, 16, 120, 64, 700, dict(nvec=4, max_iter=12, c_divisor=8, vr_period=4)),
    "k8_vr_uneven": (40, 24, 800, 64, 2600,
                     dict(nvec=8, max_iter=12, c_divisor=16, vr_period=4, cluster=4)),
}


def matrices(name):
    """Host matrices (FP32): N(0,1) entries times lognormal column scales, sizes log-uniform."""
    count, mlo, mhi, nlo, nhi, _ = BATCHES[name]
    r = np.random.default_rng(sorted(BATCHES).index(name))
    out = []
    for _ in range(count):
        m = int(round(math.exp(r.uniform(math.log(mlo), math.log(mhi)))))
        n = int(round(math.exp(r.uniform(math.log(nlo), math.log(nhi)))))
        out.append((r.standard_normal((m, n)) * np.exp(r.standard_normal(n))).astype(np.float32))
    return out


def run(name):
    """(Ritz values, iterations) of a batch on the device."""
    import torch
    from eigenvaluecomputation_by_amm_b200 import BatchSolver
    mats = []
    for A in matrices(name):
        m, n = A.shape
        buf = torch.zeros(n, (m + 3) // 4 * 4, device="cuda")
        buf[:, :m] = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
        mats.append(buf.t()[:m])
    solver = BatchSolver(mats, tol=0.0, **BATCHES[name][5])
    solver.run()
    torch.cuda.synchronize()
    out = solver.lam.cpu().numpy(), solver.iters.cpu().numpy()
    solver.close()
    return out


if __name__ == "__main__":
    sys.path.insert(0, ".")
    got = {}
    for key in BATCHES:
        got[key + "_lam"], got[key + "_iters"] = run(key)
    np.savez_compressed(sys.argv[1], **got)
