"""The single products' vectors: host memory that CUDA does not know is refused on the host (nothing is
launched and the context goes on), and vectors that are not read in place (here: off a 16-byte
boundary) give the bits of those that are, for y too."""
import ctypes as C

import numpy as np
import pytest
import torch

from helpers import scaled_gaussian, states

pytestmark = pytest.mark.gpu


def test_foreign_pointers_are_refused_and_others_copied(amm_lib):
    from eigenvaluecomputation_by_amm_b200 import AMMContext, _lib, column_major
    m, n, c = 512, 2048, 256
    ctx = AMMContext(m, n, c=c, step=1)
    ctx.set_matrix(column_major(torch.from_numpy(scaled_gaussian(m, n, seed=1)).cuda()))
    st = torch.from_numpy(states(c, 2).view(np.int32)).cuda()
    r = np.random.default_rng(3)
    host = r.standard_normal((4, m)).astype(np.float32)
    x, xm, ym = (torch.from_numpy(v).cuda() for v in host[:3])
    ctx.set_rng_state(st)
    want, _ = ctx.core_previousAMM(x, xm, ym)
    launches = amm_lib.amm_kernel_launch_count()
    at = host[3].ctypes.data
    p = [t.data_ptr() for t in (x, xm, ym)]
    y = torch.zeros(m, device="cuda")
    for args in ((at, p[1], p[2], y.data_ptr()), (p[0], at, p[2], y.data_ptr()),
                 (p[0], p[1], at, y.data_ptr()), (p[0], p[1], p[2], at)):
        assert amm_lib.amm_core_previousAMM(ctx._ctx, *args, None, None) == \
            _lib.AMM_ERR_INVALID_ARGUMENT
    assert amm_lib.amm_kernel_launch_count() == launches
    buf = torch.zeros(5, m + 1, device="cuda")
    off = [buf[i, 1 - i % 2:][:m] for i in range(4)]           # some of them 4 bytes off a boundary
    for t, v in zip(off, (x, xm, ym)):
        t.copy_(v)
    assert any(t.data_ptr() % 16 for t in off)
    ctx.set_rng_state(st)
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = amm_lib.amm_core_previousAMM(ctx._ctx, *(t.data_ptr() for t in off), None, stream)
    assert rc == _lib.AMM_OK
    assert torch.equal(off[3], want)
    ctx.close()
