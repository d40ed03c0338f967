"""The persistent step kernel's packet exchange and its two product forms on the B200, against the
oracle: shapes at the edges of the packet ownership (fewer packets than CTAs, a last packet of one
or two values, rows that do not fill the block), slices that just fit the shared-memory ring and
slices that do not, several launches per call, and an eigenvector for the error trace.

Tolerances: λ within helpers.RTOL_LAMBDA_F32, the final vector within 1e-4 (FP32 dots and partial
sums against the FP64-accumulating oracle), states and step kinds exactly.
"""
import numpy as np
import pytest
import torch

import amm_oracle as O
from helpers import RTOL_LAMBDA_F32, rel, scaled_gaussian, states, vec_rel

pytestmark = pytest.mark.gpu

# (m, n, c, dtype): 4 values per thread and fewer packets than CTAs; one more row group than a
# block of 32 threads; 8 rows per thread with idle threads (3000 BF16 rows as 375 vectors of 384);
# 16 and 32 rows per thread, full and not; a resident slice (n / 148 columns within the ring) and a
# streamed one for the same m
SHAPES = [(4, 400, 20, "f32"), (132, 300, 40, "f32"), (1024, 700, 90, "f32"),
          (1024, 9000, 500, "f32"), (2052, 1500, 150, "f32"), (8192, 900, 130, "f32"),
          (8196, 600, 77, "f32"), (16380, 700, 150, "f32"), (8, 300, 33, "bf16"),
          (3000, 2111, 301, "bf16"), (8200, 801, 99, "bf16"), (16384, 1300, 200, "bf16")]


@pytest.mark.parametrize("method,kw", [("exact", {}), ("previous", dict(vr_period=5)),
                                       ("proposed", dict(vr_period=4))])
@pytest.mark.parametrize("m,n,c,dtype", SHAPES)
def test_step_kernel_shapes(m, n, c, dtype, method, kw):
    from eigenvaluecomputation_by_amm_b200 import AMMContext, column_major
    step = 18                                      # two launches for the sampled methods
    A = scaled_gaussian(m, n, seed=m + n, shift=0.05)
    tA = torch.from_numpy(A).cuda()
    if dtype == "bf16":
        tA = tA.to(torch.bfloat16)
        A = tA.float().cpu().numpy()
    ctx = AMMContext(m, n, c=c, step=step, dtype=dtype, **kw)
    ctx.set_matrix(column_major(tA))
    st = states(c, m + c)
    ctx.set_rng_state(torch.from_numpy(st.view(np.int32)).cuda())
    x0 = np.random.default_rng(m + 5).standard_normal(m).astype(np.float32)
    vstar = np.random.default_rng(m + 6).standard_normal(m)
    vstar /= np.linalg.norm(vstar)
    ctx.set_eigenvector(torch.from_numpy(vstar))
    ctx.power_method(method, torch.from_numpy(x0).cuda())
    tr = ctx.trace()
    ref = O.power_method(A, x0, method=method, step=step, c=c, states=st, vstar=vstar, **kw)
    assert tr["kinds"] == ref.modes
    assert np.all(rel(tr["eigs"], ref.eigs) < RTOL_LAMBDA_F32), rel(tr["eigs"], ref.eigs)
    assert np.all(np.abs(tr["errs"] - ref.errs) < 1e-4)
    if method != "exact":
        assert np.array_equal(ctx.get_rng_state(c).cpu().numpy().view(np.uint32), ref.states[:c])
    x, _ = ctx.vectors()
    assert vec_rel(x.cpu().numpy(), ref.x) < 1e-4
    # the same call again: bitwise the same (fixed orders throughout, epochs that move on)
    ctx.set_rng_state(torch.from_numpy(st.view(np.int32)).cuda())
    ctx.power_method(method, torch.from_numpy(x0).cuda())
    assert np.array_equal(ctx.trace()["eigs"], tr["eigs"])
    ctx.close()


@pytest.mark.parametrize("m,n,c,dtype", [(8, 300, 33, "bf16"), (4, 400, 20, "f32"),
                                         (1024, 700, 90, "f32"), (3000, 900, 120, "bf16")])
def test_ctas_without_packets_over_many_calls(m, n, c, dtype):
    """CTAs that own no packet of y run ahead of the others; over many calls of every kind of step no
    packet is overwritten before a slower CTA has read it (the wait for it would run out and the
    call report it), and the results stay bitwise the same."""
    from eigenvaluecomputation_by_amm_b200 import AMMContext, column_major
    A = torch.from_numpy(scaled_gaussian(m, n, seed=m, shift=0.05)).cuda()
    A = A.to(torch.bfloat16) if dtype == "bf16" else A
    ctx = AMMContext(m, n, c=c, step=24, dtype=dtype, vr_period=4)
    ctx.set_matrix(column_major(A))
    st = torch.from_numpy(states(c, 3).view(np.int32)).cuda()
    x0 = torch.from_numpy(np.random.default_rng(4).standard_normal(m).astype(np.float32)).cuda()
    want = {}
    for call in range(60):
        method = ("exact", "previous", "proposed")[call % 3]
        ctx.set_rng_state(st)
        ctx.power_method(method, x0)
        eigs = ctx.trace()["eigs"]
        assert np.array_equal(eigs, want.setdefault(method, eigs))
    ctx.close()


@pytest.mark.parametrize("step", [40, 1700])
def test_trace_region_of_any_length(step):
    """A trace short enough for one copy and one that is copied piece by piece (1700 steps, stopped
    early by the tolerance) hold the same entries."""
    from eigenvaluecomputation_by_amm_b200 import AMMContext, column_major
    m, n, c = 256, 700, 90
    A = scaled_gaussian(m, n, seed=31)
    ctx = AMMContext(m, n, c=c, step=step, tol=1e-5, vr_period=4)
    ctx.set_matrix(column_major(torch.from_numpy(A).cuda()))
    st = states(c, 32)
    ctx.set_rng_state(torch.from_numpy(st.view(np.int32)).cuda())
    x0 = np.random.default_rng(33).standard_normal(m).astype(np.float32)
    ctx.power_method("exact", torch.from_numpy(x0).cuda())
    tr = ctx.trace()
    ref = O.power_method(A, x0, method="exact", step=40, c=c, states=st, vr_period=4)
    k = tr["steps_run"]
    assert 1 < k < 40
    for key in ("eigs", "errs", "coss", "distinct", "t_ns", "kinds"):
        assert len(tr[key]) == k
    assert np.all(rel(tr["eigs"], ref.eigs[:k]) < RTOL_LAMBDA_F32)
    assert np.all(np.diff(tr["t_ns"]) > 0) and set(tr["distinct"]) == {n}
    ctx.close()


@pytest.mark.parametrize("memo", ["none", "x", "both"])
def test_single_product_aligned_and_misaligned_vectors(memo):
    """A single product reads 16-byte aligned vectors in place and copies others first: the same
    result, with and without a memo pair, and with y written over an input."""
    import ctypes as C
    from eigenvaluecomputation_by_amm_b200 import AMMContext, column_major
    m, n, c = 260, 900, 80
    A = torch.from_numpy(scaled_gaussian(m, n, seed=41, shift=0.1)).cuda()
    st = torch.from_numpy(states(c, 42).view(np.int32)).cuda()
    ctx = AMMContext(m, n, c=c)
    ctx.set_matrix(column_major(A))
    g = torch.Generator(device="cuda").manual_seed(43)
    x, xm, ym = (torch.randn(m, device="cuda", generator=g) for _ in range(3))
    xm = xm if memo != "none" else None
    ym = ym if memo == "both" else None

    def product(off, over_x):
        def put(v):
            if v is None:
                return None
            buf = torch.empty(m + 4, device="cuda")
            buf[off:off + m] = v
            return buf[off:off + m]
        px, pxm, pym = put(x), put(xm), put(ym)
        y = px if over_x else torch.empty(m, device="cuda")
        ptr = lambda v: None if v is None else C.c_void_p(v.data_ptr())  # noqa: E731
        ctx.set_rng_state(st)
        rc = ctx.lib.amm_core_proposedAMM(ctx._ctx, ptr(px), ptr(pxm), ptr(pym), ptr(y), None, None)
        torch.cuda.synchronize()
        assert rc == 0
        return y.clone()

    want = product(0, False)
    assert torch.isfinite(want).all() and float(want.abs().max()) > 0
    for off, over_x in ((1, False), (0, True), (3, True)):
        assert torch.equal(product(off, over_x), want)
    ctx.close()
