"""Calls whose output is larger than L2: the grouped GEMM1 zeroes the output rows that GEMM2 adds into, or the gather pass does
(few local experts, rows with a stride of their own).  Every output starts as sevens, with sevens around it."""
import ctypes as C

import pytest
import torch

from fused_moe_b200 import _capi, synth
from fused_moe_b200 import kernel as K
from fused_moe_b200.ep import CudaOps, send_row_bytes

pytestmark = pytest.mark.gpu

T, HIDDEN, INTER = 33001, 2048, 128        # 135 MB of output, not a multiple of the CTAs


def _sevens(pad):
    """(whole buffer, its rows 1 ... T as the output)"""
    buf = torch.full((T + 2, HIDDEN + pad), 7.0, dtype=torch.bfloat16, device="cuda:0")
    return buf, buf[1:T + 1, :HIDDEN]


def _untouched_around(buf, pad):
    assert (buf[0] == 7).all() and (buf[-1] == 7).all(), "wrote outside the rows"
    assert pad == 0 or (buf[:, HIDDEN:] == 7).all(), "wrote past the rows"


def _same_up_to_sum_order(a, b):
    d = (a.float() - b.float()).abs().max().item()
    assert d <= 8 * 2.0 ** -8 * max(1.0, b.float().abs().max().item())   # order of at most eight bf16 additions


# (4, 7, 0): GEMM1 zeroes, most CTAs have no item; the others: the gather pass
@pytest.mark.parametrize("e_local,off,pad", [(4, 7, 0), (4, 7, 8), (1, 0, 8), (3, 0, 0)])
def test_rows_without_local_work_stay_zero(e_local, off, pad):
    """Few local experts, so most rows are only zeroed; and experts that no token chose, so that GEMM1 has no item."""
    dev = torch.device("cuda", 0)
    inp = synth.make_inputs(T=T, e_local=e_local, local_expert_offset=off, seed=3, hidden=HIDDEN, inter=INTER).to(dev)
    args = list(inp.args())
    buf, out = _sevens(pad)
    K.custom_kernel(*args, out=out, check_status=True)
    ws = K.get_workspace(dev, T, e_local, HIDDEN, INTER)
    ids = ws.view("topk_ids", torch.int32, (T, 8))
    none = ~((ids >= off) & (ids < off + e_local)).any(1)
    assert none.any() and (out[none] == 0).all()
    _untouched_around(buf, pad)
    assert (out[~none] != 0).any()
    # the same rows in a call small enough for the gather pass to zero them
    n = 4000
    args[0], args[2] = args[0][:n], args[2][:n]
    args[3] = args[3][:, :n].contiguous()
    _same_up_to_sum_order(out[:n], K.custom_kernel(*args))
    args = list(inp.args())
    args[1] = args[1].clone()
    args[1][off:off + e_local] = -100.0        # nobody chooses a local expert
    buf, out = _sevens(pad)
    K.custom_kernel(*args, out=out, check_status=True)
    assert (out == 0).all()
    _untouched_around(buf, pad)


def test_only_the_received_rows_are_zeroed():
    """An expert-parallel rank whose exchange could deliver more rows than L2 holds, and delivers fewer."""
    dev, lib, e_local, n = torch.device("cuda", 0), _capi.lib(), 8, 5003
    inp = synth.make_inputs(T=n, e_local=e_local, seed=4, hidden=HIDDEN, inter=INTER).to(dev)
    lg, bias, hq, hs, w1, s1, w2, s2, off, rsf = inp.args()
    want = K.custom_kernel(*inp.args(), check_status=True).clone()
    ops, stream = CudaOps(), torch.cuda.current_stream(dev).cuda_stream
    ids, w = ops.route(lg, bias, rsf, off, e_local, HIDDEN, INTER)
    sent, counts, _ = ops.pack(ids, w, hq, hs, 1)      # one rank: every token, in order
    assert counts.tolist() == [n]
    table = torch.tensor([[n, 0, 0]], dtype=torch.int32, device=dev)
    ws = K.get_workspace(dev, T, e_local, HIDDEN, INTER)
    ws.last_T = T
    buf, out = _sevens(0)
    w1b, w2b = K._as_bytes(w1, "w1"), K._as_bytes(w2, "w2")
    _capi.check(lib.b200moe_ep_local_experts(
        (C.c_void_p * 1)(sent.data_ptr()), table.data_ptr(), 1, T, send_row_bytes(HIDDEN), w1b.data_ptr(), s1.data_ptr(),
        w2b.data_ptr(), s2.data_ptr(), e_local, off, HIDDEN, INTER, ws.ptr, ws.nbytes, out.data_ptr(), HIDDEN, stream),
        "b200moe_ep_local_experts")
    assert ws.read_status(stream)[0] == 0
    _same_up_to_sum_order(out[:n], want)
    none = ~((ids >= off) & (ids < off + e_local)).any(1)
    assert none.any() and (out[:n][none] == 0).all()
    assert (out[n:] == 7).all(), "zeroed rows that nothing was received for"
    _untouched_around(buf, 0)
