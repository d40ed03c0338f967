"""The step kernel that a device with too few SMs for the packet exchange takes (grid barriers, one CTA
per SM, no clusters), asked for by AMM_PANEL_PACKETS=0 in a process of its own: the picks, step kinds
and sampling states of the packet exchange, λ within the FP32 tolerance of it and of the oracle."""
import json
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import amm_oracle as O
from helpers import RTOL_LAMBDA_F32, rel, scaled_gaussian, states

pytestmark = pytest.mark.gpu
ROOT = str(Path(__file__).resolve().parents[1])

SCRIPT = r"""
import json, sys
import numpy as np, torch
sys.path.insert(0, sys.argv[1]); sys.path.insert(0, sys.argv[1] + "/tests")
from helpers import scaled_gaussian, states
from eigenvaluecomputation_by_amm_b200 import AMMContext, column_major
out = []
for m, n, c, kw in json.loads(sys.argv[2]):
    ctx = AMMContext(m, n, c=c, step=20, **kw)
    ctx.set_matrix(column_major(torch.from_numpy(scaled_gaussian(m, n, seed=m, shift=0.05)).cuda()))
    x0 = torch.from_numpy(np.random.default_rng(m + 1).standard_normal(m).astype(np.float32)).cuda()
    for method in ("exact", "previous", "proposed"):
        ctx.set_rng_state(torch.from_numpy(states(c, m + 2).view(np.int32)).cuda())
        ctx.power_method(method, x0)
        tr = ctx.trace()
        out.append({"eigs": tr["eigs"].tolist(), "kinds": tr["kinds"],
                    "states": ctx.get_rng_state(c).cpu().numpy().view(np.uint32).tolist()})
    ctx.close()
print(json.dumps(out))
"""
CASES = [(512, 2048, 256, dict(vr_period=4)), (2052, 1500, 150, dict(vr_adaptive_threshold=1e-2)),
         (8196, 600, 77, dict(vr_period=5))]


def test_same_solves_as_with_packets(amm_lib):
    def run(extra):
        env = {k: v for k, v in os.environ.items() if not k.startswith("AMM_PANEL")}
        r = subprocess.run([sys.executable, "-c", SCRIPT, ROOT, json.dumps(CASES)],
                           env={**env, **extra}, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        return json.loads(r.stdout.strip().splitlines()[-1])

    base, got = run({}), run({"AMM_PANEL_PACKETS": "0"})
    for (m, n, c, kw), k in ((case, k) for case in CASES for k in range(3)):
        i = 3 * CASES.index((m, n, c, kw)) + k
        assert got[i]["kinds"] == base[i]["kinds"] and got[i]["states"] == base[i]["states"]
        assert np.all(rel(got[i]["eigs"], base[i]["eigs"]) < RTOL_LAMBDA_F32)
        if k == 1:
            x0 = np.random.default_rng(m + 1).standard_normal(m).astype(np.float32)
            ref = O.power_method(scaled_gaussian(m, n, seed=m, shift=0.05), x0, method="previous",
                                 step=20, c=c, states=states(c, m + 2), **kw)
            assert got[i]["kinds"] == ref.modes
            assert np.all(rel(got[i]["eigs"], ref.eigs) < RTOL_LAMBDA_F32)
    assert any(not np.array_equal(g["eigs"], b["eigs"]) for g, b in zip(got, base))  # another kernel
