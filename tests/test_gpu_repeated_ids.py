"""Ids that repeat within a token, as a caller with a router of its own may hand over: one row per (token, expert) with the
last one's weight, and no packed row without a token (the GEMM epilogues store by it)."""
import numpy as np
import pytest
import torch

from fused_moe_b200 import _capi, synth
from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu

OFF, E_LOCAL, HIDDEN, INTER = 32, 16, 512, 256


def _ids(T, seed):
    rng = np.random.default_rng(seed)
    ids = np.stack([rng.choice(np.arange(OFF - 8, OFF + E_LOCAL + 8), 8, replace=False) for _ in range(T)]).astype(np.int32)
    ids[::2, 5] = ids[::2, 1]
    ids[::3, 7] = ids[::3, 5]
    ids[T // 2] = OFF + 3                    # all eight the same
    ids[T - 1] = OFF + E_LOCAL - 1           # ... and the last token of the last expert
    return ids, rng.uniform(0.1, 1.0, (T, 8)).astype(np.float32)


# 16: the decode tile, 17 and 64: tiles of up to 64 rows, 65 and 600: the 128 x 256 tiles, more than one placement chunk
@pytest.mark.parametrize("T", [1, 16, 17, 64, 65, 600])
def test_repeated_ids_are_one_row_with_the_last_weight(T):
    lib, dev = _capi.lib(), torch.device("cuda", 0)
    inp = synth.make_inputs(T=T, e_local=E_LOCAL, local_expert_offset=OFF, seed=11, hidden=HIDDEN, inter=INTER)
    ids, w = _ids(T, T)
    once = ids.copy()                        # the same call with every expert named once
    for k in range(7):
        once[(ids[:, k + 1:] == ids[:, k:k + 1]).any(1), k] = -1
    want = O.experts_and_combine(once, w, inp.hidden_states.view(torch.uint8).numpy(), inp.hidden_states_scale.numpy(),
                                 inp.gemm1_weights.view(torch.uint8).numpy(), inp.gemm1_weights_scale.numpy(),
                                 inp.gemm2_weights.view(torch.uint8).numpy(), inp.gemm2_weights_scale.numpy(), OFF)
    want = torch.from_numpy(want.view(np.int16).copy()).view(torch.bfloat16)

    g = inp.to(dev)
    d_ids, d_w = torch.from_numpy(ids).to(dev), torch.from_numpy(w).to(dev)
    L = _capi.workspace_layout(T, E_LOCAL, HIDDEN, INTER)
    ws = torch.zeros(int(L.total_bytes), dtype=torch.uint8, device=dev)
    assert ws.data_ptr() % 256 == 0
    rows = ws[L.row_token:L.row_token + 4 * L.m_cap].view(torch.int32)
    rows.fill_(-1)                           # what the padding of earlier calls leaves behind
    out = torch.full((T + 2, HIDDEN), 7.0, dtype=torch.bfloat16, device=dev)   # a row before and one behind the output
    stream = torch.cuda.current_stream(dev).cuda_stream
    _capi.check(lib.b200moe_count(d_ids.data_ptr(), 8, T, OFF, E_LOCAL, HIDDEN, INTER, ws.data_ptr(), ws.numel(), stream),
                "b200moe_count")
    _capi.check(lib.b200moe_experts(
        d_ids.data_ptr(), 8, d_w.data_ptr(), 8, g.hidden_states.data_ptr(), g.hidden_states.stride(0),
        g.hidden_states_scale.data_ptr(), 1, T, g.gemm1_weights.data_ptr(), g.gemm1_weights_scale.data_ptr(),
        g.gemm2_weights.data_ptr(), g.gemm2_weights_scale.data_ptr(), T, E_LOCAL, OFF, HIDDEN, INTER, ws.data_ptr(),
        ws.numel(), out[1:].data_ptr(), HIDDEN, stream), "b200moe_experts")
    assert lib.b200moe_read_status(ws.data_ptr(), stream, None) == 0

    counts = ws[L.expert_count:L.expert_count + 4 * E_LOCAL].view(torch.int32).cpu().numpy()
    assert np.array_equal(counts, O.local_counts(once, OFF, E_LOCAL)), "a repeated id is counted once"
    row0 = ws[L.expert_row0:L.expert_row0 + 4 * E_LOCAL].view(torch.int32).cpu().numpy()
    tok = rows.cpu().numpy()
    for e in range(E_LOCAL):
        named = np.nonzero((once == OFF + e).any(1))[0]
        assert np.array_equal(tok[row0[e]:row0[e] + counts[e]], named), f"rows of expert {e}"
    assert (out[0] == 7).all() and (out[-1] == 7).all(), "wrote outside the output"
    frac_all, frac_nz, max_abs = synth.check_close(out[1:T + 1], want)
    assert frac_all >= 0.999 and frac_nz >= 0.999, (frac_all, frac_nz, max_abs)
