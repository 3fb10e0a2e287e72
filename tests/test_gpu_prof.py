"""B200MOE_PROF=1: CTA 0's cycle counters behind `meta`, from the streaming kernels as from the grouped ones.  The switch is read
once per process, so the calls run in a child."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import json, torch
from fused_moe_b200 import kernel, synth
dev, out = torch.device("cuda", 0), {}
for T in (7, 16, 40, 300):
    inp = synth.make_inputs(T=T, e_local=8, seed=1, zipf=True, hidden=2048, inter=512).to(dev)
    kernel.custom_kernel(*inp.args(), check_status=True)
    ws = kernel.get_workspace(dev, T, 8, 2048, 512)
    out[T] = ws.view("meta", torch.int64, (32,)).tolist()
print(json.dumps(out))
"""


def test_counters_of_both_kinds_of_gemm():
    r = subprocess.run([sys.executable, "-c", CHILD], env=dict(os.environ, B200MOE_PROF="1", PYTHONPATH=ROOT), cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    words = {int(t): w for t, w in json.loads(r.stdout.strip().splitlines()[-1]).items()}
    for T, w in words.items():
        for at in (4, 17):                     # GEMM1, GEMM2
            c = w[at:at + 10]
            assert c[9] == (1 if T <= 64 else 0), T
            assert c[3] > 0, f"{T} tokens: no K block counted"
            if T <= 64:
                wait, issue, total, _, acc, tma, mma, promo_wait, promo_total = c[:9]
                assert 0 < issue and wait + issue <= total, T
                assert acc >= 0 and tma > 0 and mma > 0, T
                assert 0 < promo_wait <= promo_total, T
            else:
                assert c[1] > 0 and c[4] >= c[1], T
