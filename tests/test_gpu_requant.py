"""The requantised codes are RNE(act / scale), bit for bit, over the whole range of fp16 activations: zeros of both signs
(a product that underflows keeps its sign), subnormals, rows of nothing but zeros (the scale's floor) and saturated rows."""
import numpy as np
import pytest
import torch

from fused_moe_b200 import synth
from oracle import moe_oracle as O
import gpu_checks

pytestmark = pytest.mark.gpu


# 7 and 16: inside the streaming GEMM1 (rows in place, rows gathered); 40 and 300: the pass behind the two kinds of GEMM1
@pytest.mark.parametrize("T", [7, 16, 40, 300])
def test_codes_over_the_range_of_fp16(T):
    e_local, hidden, inter = 8, 512, 256
    inp = synth.make_inputs(T=T, e_local=e_local, seed=2, zipf=True, hidden=hidden, inter=inter)
    # the gate rows' scales: an expert's first 128 activation columns, and the other 128
    gate = torch.tensor([[1, 1e-7], [1e-8, 1e-8], [1e-12, 1e-12], [1e7, 1], [1, 1e-5], [1e-3, 1e-8], [1e4, 1e-6], [1, 1]])
    inp.gemm1_weights_scale[:, :inter // 128] *= gate[:, :, None]
    res, ws = gpu_checks.run_gpu(inp)
    L = ws.layout_of_last_call()
    counts = ws.view("expert_count", torch.int32, (e_local,)).cpu().numpy()
    row0 = ws.view("expert_row0", torch.int32, (e_local,)).cpu().numpy()
    act = ws.view("act", torch.float16, (L.m_cap, inter)).cpu().numpy()
    act_q = ws.view("act_q", torch.uint8, (L.m_cap, inter)).cpu().numpy()
    row_scale = ws.view("row_scale", torch.float32, (L.m_cap,)).cpu().numpy()
    rows = np.concatenate([np.arange(r, r + n) for r, n in zip(row0, counts)])
    a = act[rows].astype(np.float32)
    negative_zero, top = (a == 0) & np.signbit(a), np.abs(a).max(axis=1)
    assert negative_zero.any() and (top == 0).any() and (top == 65504).any()
    assert ((a != 0) & (np.abs(a) < 2.0 ** -14)).any(), "no subnormal among the activations"
    q, s = O.requant_rows(a)
    np.testing.assert_array_equal(row_scale[rows], s)
    differ = act_q[rows] != q
    assert not differ.any(), f"{differ.sum()} codes differ, {(differ & negative_zero).sum()} of them of negative zeros"
