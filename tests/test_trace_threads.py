"""Several threads read the trace of one context at once: each gets the whole of it."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest
import torch

from helpers import scaled_gaussian, states

pytestmark = pytest.mark.gpu


def test_threads_read_one_trace(amm_lib):
    from eigenvaluecomputation_by_amm_b200 import AMMContext, column_major
    m, n, c, step = 256, 1024, 128, 60
    A = column_major(torch.from_numpy(scaled_gaussian(m, n, seed=5)).cuda())
    x0 = torch.from_numpy(np.random.default_rng(6).standard_normal(m).astype(np.float32)).cuda()
    for _ in range(5):                       # a new context each time: its first reads coincide
        ctx = AMMContext(m, n, c=c, step=step, vr_period=4)
        ctx.set_matrix(A)
        ctx.set_rng_state(torch.from_numpy(states(c, 7).view(np.int32)).cuda())
        ctx.power_method("previous", x0)
        torch.cuda.synchronize()
        with ThreadPoolExecutor(8) as pool:
            got = list(pool.map(lambda _: ctx.trace(), range(64)))
        want = ctx.trace()
        for tr in got:
            assert tr["kinds"] == want["kinds"]
            for key in ("eigs", "coss", "distinct", "t_ns"):
                if key in want:
                    assert np.array_equal(tr[key], want[key])
        ctx.close()
