"""The work that users of this package have it do, as cases that can be timed and compared.

Four kinds of case, each through the public entry points:

  solve    one power-method solve of a bound matrix: set_matrix (the one-pass set-up is part of
           an AMM solve), the sampling states, power_method, then the trace of λ and the vectors
  product  one sampled product (core_previousAMM / core_proposedAMM) on a matrix that is set up,
           as a host-driven loop calls it once per step
  batch    one run of a BatchSolver over many uneven matrices
  grad     λ_max of a batch of matrices with its gradient (forward and backward)

λ is the FP64 Rayleigh quotient of FP32 products; it is returned in FP32, the type of the
products it comes from.
"""
import math

import numpy as np
import torch

from eigenvaluecomputation_by_amm_b200 import AMMContext, BatchSolver
from eigenvaluecomputation_by_amm_b200.autograd import lambda_max

ON_CHIP = 100e6  # bytes: a matrix below this need not be read from memory once per step


def _solve(name, method, m, n, c, step, vr_period=0, dtype="f32", data="scaled"):
    d = {"kind": "solve", "method": method, "m": m, "n": n, "c": c, "step": step,
         "vr_period": vr_period, "dtype": dtype, "data": data}
    return dict(d, name=name) if name else d


def _batch(name, count, mlo, mhi, nlo, nhi, nvec, products, c_divisor=0, vr_period=0):
    d = {"kind": "batch", "count": count, "mlo": mlo, "mhi": mhi, "nlo": nlo, "nhi": nhi,
         "nvec": nvec, "products": products, "c_divisor": c_divisor, "vr_period": vr_period}
    return dict(d, name=name) if name else d


def listed():
    return [
        # the smallest solve: a matrix of about a megabyte, a few AMM steps; latency and launches
        _solve("previous_f32_256x1024", "previous", 256, 1024, 128, 8, vr_period=3),
        # the size of the reference's CPU check, solved exactly (A stays on the chip)
        _solve("exact_f32_1024x4096", "exact", 1024, 4096, 0, 24),
        # the eigenfaces comparison: many cheap sampled steps on 64 x 64 images
        _solve("previous_f32_4096x16384_faces", "previous", 4096, 16384, 1024, 300, data="faces"),
        # one sampled product of a host-driven loop at the same size
        {"name": "product_proposed_f32_4096x16384", "kind": "product", "method": "proposed",
         "m": 4096, "n": 16384, "c": 1024, "dtype": "f32", "data": "scaled"},
        # two-phase driver, BF16, sizes that divide nothing (rows not filling a block, odd n)
        _solve("v2_bf16_3000x10007", "proposed_v2", 3000, 10007, 701, 30, vr_period=6,
               dtype="bf16"),
        # the exact method on the largest square FP32 matrix (1 GiB), the reference's own form
        _solve("exact_f32_16384x16384", "exact", 16384, 16384, 0, 6),
        # the headline: time to λ by proposed AMM on a 2 GiB BF16 matrix, set-up included
        _solve("proposed_bf16_16384x65536", "proposed", 16384, 65536, 4096, 9, vr_period=8,
               dtype="bf16", data="spiked"),
        # hundreds of uneven matrices, exact block products (8 vectors)
        _batch("batch_exact_512", 512, 64, 2048, 256, 8192, 8, 20),
        # the same with sampled products and variance reduction
        _batch("batch_vr_512", 512, 64, 2048, 256, 8192, 8, 20, c_divisor=8, vr_period=4),
        # a few small matrices, 4 vectors: launch cost and the per-step fixed cost
        _batch("batch_exact_24_small", 24, 24, 200, 60, 900, 4, 12),
        # the differentiation batch: forward and backward
        {"name": "grad_64x512x2048", "kind": "grad", "B": 64, "m": 512, "n": 2048, "tol": 1e-6},
        # tall matrices of a training step (solved in place as the transposed problem)
        {"name": "grad_16x700x300", "kind": "grad", "B": 16, "m": 700, "n": 300, "tol": 1e-6},
    ]


def _log_int(rng, lo, hi, multiple=1):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(multiple, v // multiple * multiple)


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "product", "batch", "batch", "grad"])
    if kind in ("solve", "product"):
        dtype = rng.choice(["f32", "bf16"])
        m = _log_int(rng, 128, 16384, 8)
        n = _log_int(rng, 512, 65536 if dtype == "bf16" else 32768)
        c = max(16, n // rng.randint(4, 24))
        if kind == "product":
            return {"kind": "product", "method": rng.choice(["previous", "proposed"]), "m": m,
                    "n": n, "c": c, "dtype": dtype, "data": "scaled"}
        method = rng.choice(["exact", "previous", "proposed", "proposed_v2"])
        step = rng.randint(6, 12) if m * n > 2 ** 27 else rng.randint(8, 60)
        return _solve(None, method, m, n, 0 if method == "exact" else c, step,
                      vr_period=rng.randint(3, min(step, 8)), dtype=dtype,
                      data=rng.choice(["scaled", "spiked"]))
    if kind == "batch":
        mhi, nhi = _log_int(rng, 100, 2048), _log_int(rng, 400, 8192)
        sampled = rng.random() < 0.4
        return _batch(None, _log_int(rng, 8, 300), max(16, mhi // 16), mhi, max(64, nhi // 16),
                      nhi, rng.choice([4, 8, 8]), rng.randint(8, 20),
                      c_divisor=8 if sampled else 0, vr_period=4 if sampled else 0)
    return {"kind": "grad", "B": _log_int(rng, 4, 64), "m": _log_int(rng, 48, 800, 4),
            "n": _log_int(rng, 48, 1600, 4), "tol": 1e-6}


# ---- inputs ----
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _matrix(case, seed):
    """(n, m) row-major storage of A, i.e. A column-major: N(0,1) entries times lognormal column
    scales; "spiked" adds 30·u·wᵀ (u, w unit); "faces": mean-centred mixtures of smooth patterns."""
    m, n, g = case["m"], case["n"], _gen(seed)
    if case["data"] == "faces":
        side = int(math.isqrt(m))
        i = (torch.arange(side, device="cuda") + 0.5) / side
        f = torch.arange(8, device="cuda")
        cosines = torch.cos(math.pi * f[:, None] * i[None, :])
        P = torch.einsum("ai,bj->abij", cosines, cosines).reshape(64, m)[1:51]
        P = P / P.norm(dim=1, keepdim=True)
        k = torch.arange(1, 51, device="cuda")
        At = (torch.randn(n, 50, device="cuda", generator=g) * k ** -0.75) @ P
        At += 0.02 * torch.randn(n, m, device="cuda", generator=g)
        At -= At.mean(dim=1, keepdim=True)
        At *= torch.exp(0.5 * torch.randn(n, 1, device="cuda", generator=g))
        return At
    wanted = torch.float32 if case["dtype"] == "f32" else torch.bfloat16
    scale = torch.exp(torch.randn(n, 1, device="cuda", generator=g))
    u = torch.randn(m, device="cuda", generator=g)
    w = torch.randn(n, device="cuda", generator=g)
    u, w = 30.0 * u / u.norm(), w / w.norm()
    At = torch.empty(n, m, dtype=wanted, device="cuda")
    for lo in range(0, n, 8192):
        blk = torch.randn(min(8192, n - lo), m, device="cuda", generator=g) * scale[lo:lo + 8192]
        if case["data"] == "spiked":
            blk += w[lo:lo + 8192, None] * u[None, :]
        At[lo:lo + 8192] = blk.to(wanted)
    return At


def _states(count, seed):
    r = np.random.default_rng(seed)
    return r.integers(1, 2 ** 32, size=count, dtype=np.uint64).astype(np.uint32)


def _shapes(case, seed):
    r = np.random.default_rng(seed)
    ln = lambda lo, hi: int(round(math.exp(r.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    return [(ln(case["mlo"], case["mhi"]), ln(case["nlo"], case["nhi"]))
            for _ in range(case["count"])]


def _batch_matrices(case, seed):
    """Column-major FP32 matrices (leading dimension: rows rounded up to 4).  The shapes are the
    case's own, the values the seed's."""
    mats, g = [], _gen(seed)
    for m, n in _shapes(case, 7):
        buf = torch.zeros(n, (m + 3) // 4 * 4, device="cuda")
        buf[:, :m] = torch.randn(n, m, device="cuda", generator=g) * torch.exp(
            torch.randn(n, 1, device="cuda", generator=g))
        mats.append(buf.t()[:m])
    return mats


def _grad_input(case, seed):
    g = _gen(seed)
    A = torch.randn(case["B"], case["m"], case["n"], device="cuda", generator=g)
    A *= torch.exp(0.5 * torch.randn(case["B"], 1, case["n"], device="cuda", generator=g))
    return A


def prepare(case, seed):
    if case["kind"] == "batch":
        mats = _batch_matrices(case, seed)
        return case, BatchSolver(mats, nvec=case["nvec"], max_iter=case["products"], tol=0.0,
                                 c_divisor=case["c_divisor"], vr_period=case["vr_period"])
    if case["kind"] == "grad":
        return case, _grad_input(case, seed)
    A = _matrix(case, seed).t()
    m, n, c = case["m"], case["n"], case["c"] or case["n"]
    x0 = torch.randn(m, device="cuda", generator=_gen(seed + 1))
    st = torch.from_numpy(_states(c, seed).view(np.int32)).cuda()
    ctx = AMMContext(m, n, c=c, step=case.get("step", 1), vr_period=case.get("vr_period", 0),
                     dtype=case["dtype"])
    if case["kind"] == "product":
        ctx.set_matrix(A)
        xm = x0 + 0.1 * x0.norm() / math.sqrt(m) * torch.randn(m, device="cuda",
                                                              generator=_gen(seed + 2))
        return case, ctx, A, st, x0 / x0.norm(), xm / xm.norm(), ctx.exact_product(xm / xm.norm())
    return case, ctx, A, st, x0


def run(state):
    case = state[0]
    if case["kind"] == "batch":
        solver = state[1]
        solver.run()
        return {"lam": solver.lam.float(), "vectors": solver.vectors, "iters": solver.iters}
    if case["kind"] == "grad":
        A = state[1].detach().requires_grad_(True)
        lam = lambda_max(A, tol=case["tol"])
        lam.sum().backward()
        return {"lam": lam.detach().float(), "grad": A.grad}
    if case["kind"] == "product":
        _, ctx, _, st, x, xm, ym = state
        ctx.set_rng_state(st)
        product = ctx.core_previousAMM if case["method"] == "previous" else ctx.core_proposedAMM
        y, idx = product(x, xm, ym)
        return {"y": y, "idx": idx}
    _, ctx, A, st, x0 = state
    ctx.set_matrix(A)
    if case["method"] != "exact":
        ctx.set_rng_state(st)
    ctx.power_method(case["method"], x0)
    tr = ctx.trace()
    x, y = ctx.vectors()
    return {"lam": tr["eigs"].astype(np.float32), "cos": tr["coss"].astype(np.float32),
            "distinct": tr["distinct"], "x": x, "y": y}


# ---- the work that cannot be done without ----
def _kinds(case):
    """Kind of every step of a solve: True for the steps that read every column."""
    vr, le, out = case["vr_period"], 0, []
    for i in range(case["step"]):
        periodic = vr > 0 and (i + 1) % vr == 0
        if case["method"] == "exact":
            out.append("exact")
        elif case["method"] == "previous":
            out.append("memo" if periodic else "previous")
        elif case["method"] == "proposed":
            memo = periodic and i > le + 1
            le = i if memo else le
            out.append("memo" if memo else "proposed")
        else:
            out.append("previous" if i < vr - 1 else "exact" if i == vr - 1
                       else "memo" if periodic else "proposed")
    return out


def work(case):
    if case["kind"] == "batch":
        el = sum(m * n for m, n in _shapes(case, 7))
        p, vr = case["products"], case["vr_period"]
        if case["c_divisor"]:
            full = sum(1 for i in range(p) if vr and ((i + 1) % vr == 0 or i + 1 >= p))
            p = full + (p - full) / case["c_divisor"]
        return {"bytes": 4.0 * el, "flops": 4.0 * el * p * case["nvec"]}
    if case["kind"] == "grad":
        el = case["B"] * case["m"] * case["n"]
        return {"bytes": 8.0 * el, "flops": 4.0 * el * 8 * 10}
    m, n, es = case["m"], case["n"], 4 if case["dtype"] == "f32" else 2
    distinct = n * (1 - (1 - 1 / n) ** (case["c"] or n))
    if case["kind"] == "product":
        return {"bytes": distinct * m * es + 16.0 * m, "flops": 4.0 * distinct * m}
    kinds = _kinds(case)
    full = sum(k in ("exact", "memo") for k in kinds)
    cols = full * n + (len(kinds) - full) * distinct
    if m * n * es < ON_CHIP:
        read = n
    else:
        read = cols + (0 if case["method"] == "exact" else n)
    return {"bytes": float(read * m * es + 16 * m), "flops": 4.0 * cols * m}


# ---- the same results in 64 bits ----
class _Columns:
    """Blocks of columns of A (given as (n, m) storage) in FP64."""

    def __init__(self, At):
        self.At = At

    def __iter__(self):
        step = max(1, 2 ** 27 // self.At.shape[1])
        for lo in range(0, self.At.shape[0], step):
            yield lo, self.At[lo:lo + step].double()

    def stats(self):
        s = torch.zeros(self.At.shape[0], dtype=torch.float64, device="cuda")
        q, z = s.clone(), torch.zeros(self.At.shape[1], dtype=torch.float64, device="cuda")
        m = self.At.shape[1]
        for lo, b in self:
            s[lo:lo + len(b)], q[lo:lo + len(b)] = b.sum(1), (b * b).sum(1)
            z += (b.sum(1) / m) @ b
        alpha = s / m
        return (alpha, q.sqrt().float().double(),
                (q - alpha * alpha * m).clamp(min=0).sqrt().float().double(), z)

    def exact(self, x):
        return sum((b @ x) @ b for _, b in self)


def _draw(states, cdf):
    """One xorshift32 step of every state and the columns that the inverse CDF picks."""
    y = states
    y = y ^ (y << np.uint32(13))
    y = y ^ (y >> np.uint32(17))
    y = y ^ (y << np.uint32(5))
    u = (y & np.uint32(0x7FFFFF)).astype(np.float64) / 2.0 ** 23
    target = cdf[-1] * torch.from_numpy(u).cuda()
    return y, torch.searchsorted(cdf, target, right=True).clamp(max=len(cdf) - 1)


def _sampled(At, stats, centred, picks, c, dx, ym):
    alpha, norm, normp, z = stats
    w2 = (normp if centred else norm) ** 2
    cols, mult = torch.unique(picks, return_counts=True)
    w = w2.sum() / (w2[cols] * c) * mult
    S = At[cols].double()
    t = (S @ dx - (alpha[cols] * dx.sum() if centred else 0.0)) * w
    y = ym + t @ S
    if centred:
        y = y + dx.sum() * (z - (alpha * alpha).sum()) + z @ dx - (alpha[cols] * t).sum()
    return y, len(cols)


def _exact_solve(case, seed):
    At = _matrix(case, seed)
    m, c = case["m"], case["c"] or case["n"]
    x0 = torch.randn(m, device="cuda", generator=_gen(seed + 1))
    cols, st = _Columns(At), _states(c, seed)
    x = x0.double() / x0.double().norm()
    if case["method"] != "exact":
        stats = cols.stats()
        cdf = [torch.cumsum(stats[k] ** 2, 0) for k in (1, 2)]
    xm = ym = torch.zeros(m, dtype=torch.float64, device="cuda")
    lam, cos = [], []
    for kind in _kinds(case):
        if kind in ("exact", "memo"):
            y = cols.exact(x)
            if kind == "memo":
                xm, ym = x, y
        else:
            centred = kind == "proposed"
            st, picks = _draw(st, cdf[1 if centred else 0])
            y, _ = _sampled(At, stats, centred, picks, c, x - xm, ym)
        lam.append(float(x @ y))
        cos.append(float(x @ y / y.norm()))
        x = y / y.norm()
    return {"lam": np.array(lam), "cos": np.array(cos), "distinct": None, "x": x, "y": y}


def _exact_product(case, seed):
    At = _matrix(case, seed)
    m, c = case["m"], case["c"]
    x0 = torch.randn(m, device="cuda", generator=_gen(seed + 1))
    xm = x0 + 0.1 * x0.norm() / math.sqrt(m) * torch.randn(m, device="cuda",
                                                          generator=_gen(seed + 2))
    x, xm = (x0 / x0.norm()).double(), (xm / xm.norm()).double()
    cols = _Columns(At)
    stats, centred = cols.stats(), case["method"] == "proposed"
    _, picks = _draw(_states(c, seed), torch.cumsum(stats[2 if centred else 1] ** 2, 0))
    y, _ = _sampled(At, stats, centred, picks, c, x - xm, cols.exact(xm))
    return {"y": y, "idx": None}


def _start_block(b, m, nvec, seed=1234):
    """The start block of matrix b: a counter-based hash of (seed, matrix, row, vector)."""
    g, mask = 0x9E3779B97F4A7C15, 2 ** 64 - 1
    row = np.arange(m, dtype=np.uint64)[:, None]
    vec = np.arange(nvec, dtype=np.uint64)[None, :]
    z = np.uint64(seed ^ (g * (b + 1) & mask)) ^ (row << np.uint64(20)) ^ (vec << np.uint64(52))
    z = z + np.uint64(g)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    z = z ^ (z >> np.uint64(31))
    v = (z >> np.uint64(32)).astype(np.uint32).view(np.int32).astype(np.float64) / 2.0 ** 31
    return torch.from_numpy(v).cuda()


def _exact_batch(case, seed):
    """Ritz values of the block after the products, every product exact."""
    out = []
    for b, A in enumerate(_batch_matrices(case, seed)):
        A = A.double()
        X = torch.linalg.qr(_start_block(b, A.shape[0], case["nvec"]))[0]
        for _ in range(case["products"]):
            Y = A @ (A.t() @ X)
            H = X.t() @ Y
            L = torch.linalg.cholesky_ex(Y.t() @ Y)[0]
            X = torch.linalg.solve_triangular(L, Y.t(), upper=False).t()
        out.append((H + H.t()) / 2)
    lam = torch.linalg.eigvalsh(torch.stack(out)).flip(1)
    return {"lam": lam, "vectors": None, "iters": None}


def _exact_grad(case, seed):
    A = _grad_input(case, seed).double()
    tall = case["m"] > case["n"]
    w, V = torch.linalg.eigh(A.transpose(1, 2) @ A if tall else A @ A.transpose(1, 2))
    v = V[:, :, -1:]
    grad = 2.0 * ((A @ v) @ v.transpose(1, 2) if tall else v @ (v.transpose(1, 2) @ A))
    return {"lam": w[:, -1], "grad": grad}


def exact(case, seed):
    return {"solve": _exact_solve, "product": _exact_product, "batch": _exact_batch,
            "grad": _exact_grad}[case["kind"]](case, seed)
