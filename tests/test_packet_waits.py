"""The step kernel's packet waits are bounded: waiting for an epoch that nothing writes, each of their
three forms gives up after 2 s, the host reads AMM_ERR_DEVICE_TIMEOUT, and the context then solves."""
import ctypes as C

import numpy as np
import pytest
import torch

from helpers import scaled_gaussian

pytestmark = pytest.mark.gpu


def test_packet_waits_give_up(amm_lib):
    from eigenvaluecomputation_by_amm_b200 import AMMContext, _lib, column_major
    ctx = AMMContext(256, 1024, c=128, step=6)
    ctx.set_matrix(column_major(torch.from_numpy(scaled_gaussian(256, 1024, seed=4)).cuda()))
    x0 = torch.ones(256, device="cuda")
    ctx.power_method("exact", x0)
    want = ctx.trace()["eigs"]
    out = (C.c_uint32 * 3)()
    assert amm_lib.amm_probe_bounded_waits(ctx._ctx, out, None) == _lib.AMM_ERR_DEVICE_TIMEOUT
    assert out[0] == 0 and out[1] == 0
    assert 9.9e6 <= out[2] <= 30e6            # five waits of 2 s, in µs
    ctx.power_method("exact", x0)
    assert np.array_equal(ctx.trace()["eigs"], want)
    ctx.close()
