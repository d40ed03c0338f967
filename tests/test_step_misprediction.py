"""Adaptive variance reduction: the kind of a step depends on the cosine of the one before, so the list
whose first columns the step kernel copies ahead can be the wrong one.  Shapes at which the wrong list
fills the shared-memory ring: all n columns predicted where a sampled step follows (n/148 columns a
CTA), and a sampled list predicted where an exact step follows, which fits the ring or does not.

Tolerances: λ within helpers.RTOL_LAMBDA_F32 of the oracle, the final vector within 1e-4, step kinds
exactly (the cosines lie 2e-4 and more from the threshold), the same call again bitwise the same.
"""
import numpy as np
import pytest
import torch

import amm_oracle as O
from helpers import RTOL_LAMBDA_F32, rel, scaled_gaussian, states, vec_rel

pytestmark = pytest.mark.gpu

# (m, n, c, dtype, seed, threshold, exact steps followed by sampled ones): 44, 10, 3 and 6 columns a
# CTA; then sampled lists of 45 and 9.5
CASES = [(1024, 6512, 500, "f32", 1, 0.04, True), (4096, 1480, 200, "f32", 2, 2e-3, True),
         (16384, 444, 120, "f32", 0, 5e-3, True), (16384, 888, 200, "bf16", 3, 2e-3, True),
         (1024, 16000, 44000, "f32", 0, 0.1, False), (4096, 4000, 6500, "f32", 0, 0.1, False)]


@pytest.mark.parametrize("m,n,c,dtype,seed,thr,back", CASES)
def test_wrong_list_copied_ahead(m, n, c, dtype, seed, thr, back):
    from eigenvaluecomputation_by_amm_b200 import AMMContext, column_major
    step = 14
    A = scaled_gaussian(m, n, seed=m + n + seed, shift=0.05)
    tA = torch.from_numpy(A).cuda()
    if dtype == "bf16":
        tA = tA.to(torch.bfloat16)
        A = tA.float().cpu().numpy()
    st = states(c, m + c)
    x0 = np.random.default_rng(m + 5).standard_normal(m).astype(np.float32)
    ref = O.power_method(A, x0, method="previous", step=step, c=c, states=st,
                         vr_adaptive_threshold=thr)
    assert np.min(np.abs(ref.coss - (1 - thr))) > 2e-4
    kinds = ["exact" if k == "exact" else "sampled" for k in ref.modes]
    turns = set(zip(kinds, kinds[1:]))
    assert ("sampled", "exact") in turns and (("exact", "sampled") in turns) == back
    ctx = AMMContext(m, n, c=c, step=step, dtype=dtype, vr_adaptive_threshold=thr)
    ctx.set_matrix(column_major(tA))
    first = None
    for _ in range(20):
        ctx.set_rng_state(torch.from_numpy(st.view(np.int32)).cuda())
        ctx.power_method("previous", torch.from_numpy(x0).cuda())
        tr = ctx.trace()
        assert tr["kinds"] == ref.modes
        assert np.all(rel(tr["eigs"], ref.eigs) < RTOL_LAMBDA_F32), rel(tr["eigs"], ref.eigs)
        x, _ = ctx.vectors()
        assert vec_rel(x.cpu().numpy(), ref.x) < 1e-4
        first = tr["eigs"] if first is None else first
        assert np.array_equal(tr["eigs"], first)
    ctx.close()
