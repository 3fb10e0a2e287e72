"""Calls whose output is larger than L2: the grouped GEMM1 zeroes the output rows that GEMM2 adds into."""
import pytest
import torch

from fused_moe_b200 import kernel as K
from fused_moe_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e_local,off", [(1, 0), (4, 7)])
def test_rows_without_local_work_stay_zero(e_local, off):
    """Few local experts, so most rows are only zeroed; and an expert that no token chose, so that GEMM1 has no item."""
    dev = torch.device("cuda", 0)
    T, hidden, inter = 33001, 2048, 128        # 135 MB of output, not a multiple of the CTAs
    inp = synth.make_inputs(T=T, e_local=e_local, local_expert_offset=off, seed=3, hidden=hidden, inter=inter).to(dev)
    args = list(inp.args())
    out = torch.full((T, hidden + 8), 7.0, dtype=torch.bfloat16, device=dev)   # a row stride of its own
    K.custom_kernel(*args, out=out[:, :hidden], check_status=True)
    ws = K.get_workspace(dev, T, e_local, hidden, inter)
    ids = ws.view("topk_ids", torch.int32, (T, 8))
    none = ~((ids >= off) & (ids < off + e_local)).any(1)
    assert none.any() and (out[none][:, :hidden] == 0).all()
    assert (out[:, hidden:] == 7).all(), "wrote past the rows"
    assert (out[~none][:, :hidden] != 0).any()
    # the same rows in a call small enough for the gather pass to zero them
    n = 4000
    args[0], args[2] = args[0][:n], args[2][:n]
    args[3] = args[3][:, :n].contiguous()
    small = K.custom_kernel(*args)
    d = (small.float() - out[:n, :hidden].float()).abs().max().item()
    assert d <= 8 * 2.0 ** -8 * max(1.0, small.float().abs().max().item())   # order of at most eight bf16 additions
    args[1] = args[1].clone()
    args[1][off:off + e_local] = -100.0        # nobody chooses a local expert
    big = list(inp.args())
    big[1] = args[1]
    assert (K.custom_kernel(*big, check_status=True) == 0).all()
