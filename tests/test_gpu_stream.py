"""The weight-streaming GEMMs (decode and calls of at most 64 tokens) at the edges of their tiles: token rows around 16, 32
and 64 per expert, K ranges that are one K block, an odd number of K blocks and many, cut and uncut ranges."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT
from fused_moe_b200 import synth
import gpu_checks

pytestmark = pytest.mark.gpu


# hidden / 128 is the number of K blocks of GEMM1, inter / 128 of GEMM2; the Zipf bias gives a few experts all tokens
@pytest.mark.parametrize("T,e_local,off,zipf,hidden,inter", [
    (1, 32, 0, True, 256, 128),       # one row per expert, GEMM2 of a single K block
    (2, 256, 0, False, 512, 384),     # more slabs than SMs, odd K in GEMM2
    (8, 32, 0, True, 1024, 640),      # rows fetched in place, whole tiles of eight
    (9, 32, 0, True, 1024, 384),      # the first size with a gather pass
    (15, 8, 0, True, 2048, 256),
    (8, 32, 0, True, 8192, 128),      # the most K blocks, rows in place and gathered
    (16, 32, 0, True, 8192, 128),
    (16, 32, 0, True, 256, 896),      # a full 16-row tile, K ranges of one group
    (17, 32, 0, True, 512, 128),      # one row past it: 32-row boxes
    (32, 16, 0, True, 256, 384),
    (33, 32, 0, True, 1024, 128),     # 64-row boxes
    (64, 64, 0, True, 512, 640),      # a full 64-row tile, the most experts
    (64, 32, 224, False, 768, 384),
])
def test_stage_by_stage(T, e_local, off, zipf, hidden, inter):
    inp = synth.make_inputs(T=T, e_local=e_local, local_expert_offset=off, seed=5, zipf=zipf, hidden=hidden, inter=inter)
    res, ws = gpu_checks.run_gpu(inp)
    gpu_checks.check_stages(inp, res, ws, verbose=True)


@pytest.mark.parametrize("switch", ["B200MOE_DECODE", "B200MOE_STREAM"])
def test_switched_off(switch):
    """The switches are read once per process: the cases above on the 128 x 256 tiles (B200MOE_DECODE=0: up to 16 tokens;
    B200MOE_STREAM=0: 17 to 64)."""
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-k", "stage_by_stage",
                        os.path.join(ROOT, "tests", "test_gpu_stream.py")],
                       env=dict(os.environ, **{switch: "0"}), cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]
    assert "passed" in r.stdout
