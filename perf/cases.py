"""The workloads whose speed counts, as a user's program runs them on one GPU.

A case is one call of the fused MoE layer (DeepSeek-V3 shape: hidden 7168, intermediate 2048, 256 routed experts,
top-8) through ``fused_moe_b200.kernel``, or the device work of one rank's expert-parallel step.  Sizes are those
of the repository's configurations, benchmark and tests: the 32-expert slice at the contest's token counts
(1 ... 14107), the whole 256-expert layer that a single GPU serves, the Zipf stress, and 4096 tokens per rank.

Fields of a case:
  tokens      tokens of the call (of every rank, for an expert-parallel step)
  experts     local experts; ``offset`` is the first one's global id
  logits      "fp32" or "bf16" routing logits
  scales      "kt": hidden_states_scale [K/128, T] (contest layout), "tk": [T, K/128]
  zipf        routing bias of the load-imbalance stress instead of N(0, 0.1)
  dispatched  every token has chosen at least one local expert, as an expert-parallel rank receives them
  own_out     the caller passes its own output tensor (an engine's destination), else the module's buffer
  world       > 0: device work of one rank in a step over so many ranks (route, pack, local experts, combine)
"""
import ctypes
import math

import torch

from fused_moe_b200 import _capi, ep, kernel, synth

HIDDEN, INTER, RSF = synth.HIDDEN, synth.INTER, 2.5


def _case(name, tokens, experts, offset=0, logits="fp32", scales="kt", zipf=False, dispatched=False, own_out=False,
          world=0):
    c = dict(tokens=tokens, experts=experts, offset=offset, logits=logits, scales=scales, zipf=zipf,
             dispatched=dispatched, own_out=own_out, world=world)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one user's decode step on a slice: the latency floor of a call
        _case("slice_t1", 1, 32, dispatched=True),
        # a contest decode batch, odd size, on another rank's experts
        _case("slice_t7", 7, 32, offset=96),
        # decode batch that an engine hands over as bf16 logits with its own destination
        _case("slice_t16", 16, 32, offset=32, logits="bf16", dispatched=True, own_out=True),
        # mid-size contest batches: the square scale tensor, then past one warp tile and ragged
        _case("slice_t56", 56, 32),
        _case("slice_t80", 80, 32, offset=224, logits="bf16"),
        # the whole layer on one GPU: a small decode batch reaches most of the experts' weights
        _case("layer_t4", 4, 256, own_out=True),
        _case("layer_t64", 64, 256),
        # prefill on a slice: ragged chunk, scales laid out per token, and the largest contest batch
        _case("slice_t901", 901, 32, logits="bf16", scales="tk"),
        _case("slice_t14107", 14107, 32),
        # load imbalance: a handful of experts take every token
        _case("slice_zipf_t2048", 2048, 32, zipf=True),
        # the benchmark's step on one GPU
        _case("layer_t4096", 4096, 256),
        # one rank's device work in an 8-rank step
        _case("ep8_rank_t1024", 1024, 32, offset=64, world=8),
    ]


def draw(rng):
    """One more case: the kinds of ``listed()`` over their whole ranges."""
    kind = rng.choice(["slice", "slice", "slice", "layer", "part", "zipf", "ep"])
    experts = {"slice": 32, "zipf": 32, "layer": 256, "part": rng.choice([64, 128]), "ep": 0}[kind]
    lo, hi = {"slice": (1, 16384), "zipf": (64, 3072), "layer": (1, 3600), "part": (1, 4096), "ep": (64, 2048)}[kind]
    tokens = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if kind == "ep":
        world = rng.choice([4, 8])
        return _case("", tokens, 256 // world, offset=256 // world * rng.randrange(world), world=world)
    dispatched = tokens <= 64 and experts < 256 and rng.random() < 0.5
    return _case("", tokens, experts, offset=0 if kind == "zipf" else experts * rng.randrange(256 // experts),
                 logits=rng.choice(["fp32", "bf16"]), scales=rng.choice(["kt", "kt", "tk"]), zipf=kind == "zipf",
                 dispatched=dispatched or (tokens < 8 and experts < 256), own_out=rng.random() < 0.5)


def _route(logits, bias):
    """Expert ids [T, 8] of the no-aux routing (torch; for choosing and counting tokens only)."""
    s = logits.float().sigmoid() + bias.float()
    top2 = s.view(-1, 8, 32).topk(2, dim=-1).values.sum(-1)
    keep = torch.zeros_like(top2).scatter_(1, top2.topk(4, dim=-1).indices, 1.0)
    return s.masked_fill(keep.repeat_interleave(32, dim=1) == 0, -math.inf).topk(8, dim=-1).indices


def _local(ids, case):
    return (ids >= case["offset"]) & (ids < case["offset"] + case["experts"])


def _logits(tokens, bias, case, g, dev):
    n = tokens * 64 + 256 if case["dispatched"] else tokens
    lg = torch.randn(n, 256, generator=g, device=dev)
    if case["logits"] == "bf16":
        lg = lg.to(torch.bfloat16)
    if case["dispatched"]:
        lg = lg[_local(_route(lg, bias), case).any(1)]
        if lg.shape[0] < tokens:    # a slice that the bias starves: its few tokens come again
            lg = lg.repeat(-(-tokens // max(lg.shape[0], 1)), 1)
        lg = lg[:tokens].contiguous()
    return lg


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(1000003 * seed + 17)
    T = case["tokens"]
    bias = synth.make_bias(seed % 9973, case["zipf"]).to(dev)
    weights = synth.make_weights(case["experts"], case["offset"], seed % 99991, device=dev, fast_device_rng=True)

    def tokens():
        lg = _logits(T, bias, case, g, dev)
        hq, hs = synth.quant_rows_1x128(torch.randn(T, HIDDEN, generator=g, device=dev))
        return lg, hq, hs if case["scales"] == "kt" else hs.t().contiguous()

    st = {"case": case, "bias": bias, "w": weights}
    if case["world"]:
        # what the other ranks of the step have packed and computed, in buffers that this rank can read
        world, ops = case["world"], ep.CudaOps()
        rank = case["offset"] // case["experts"]
        rb = ep.send_row_bytes(HIDDEN)
        sent, table = [], []
        for r in range(world):
            lg, hq, hs = tokens()
            ids, w = ops.route(lg, bias, RSF, case["offset"], case["experts"], HIDDEN, INTER)
            buf = torch.zeros((4 * T, rb), dtype=torch.uint8, device=dev)
            rows, counts, slot = ops.pack(ids, w, hq, hs, world, send_buffer=buf)
            sent.append(buf)
            n = counts.tolist()
            table.append([n[rank], sum(n[:rank]), 0])
            if r == rank:
                st["mine"], st["send"] = (lg, hq, hs), buf
                starts = torch.tensor([0] * world, dtype=torch.int32, device=dev)
        st["partials"] = [torch.randn(T, HIDDEN, generator=g, device=dev).to(torch.bfloat16) for _ in range(world)]
        st["starts"], st["sent"] = starts, sent
        st["table"] = torch.tensor(table, dtype=torch.int32, device=dev)
        st["rows_out"] = torch.zeros((world * T, HIDDEN), dtype=torch.bfloat16, device=dev)   # rows past the received: 0
        return st
    st["tokens"] = tokens()
    st["out"] = torch.empty((T, HIDDEN), dtype=torch.bfloat16, device=dev) if case["own_out"] else None
    return st


def _run_rank(st):
    """The device work of one rank of an expert-parallel step (``ep.ExpertParallelMoE``, ranks that read each
    other's buffers in place), without the two small collectives between its parts."""
    case, (lg, hq, hs), ops = st["case"], st["mine"], ep.CudaOps()
    T, world, experts, offset = case["tokens"], case["world"], case["experts"], case["offset"]
    w1, s1, w2, s2 = st["w"]
    dev, lib = lg.device, _capi.lib()
    ids, w = ops.route(lg, st["bias"], RSF, offset, experts, HIDDEN, INTER)
    _, counts, slot = ops.pack(ids, w, hq, hs, world, send_buffer=st["send"])
    cap = world * T
    ws = kernel.get_workspace(dev, cap, experts, HIDDEN, INTER)
    ws.last_T = cap
    stream = torch.cuda.current_stream(dev).cuda_stream
    bases = (ctypes.c_void_p * world)(*[b.data_ptr() for b in st["sent"]])
    _capi.check(lib.b200moe_ep_local_experts(
        bases, st["table"].data_ptr(), world, cap, ep.send_row_bytes(HIDDEN), w1.data_ptr(), s1.data_ptr(),
        w2.data_ptr(), s2.data_ptr(), experts, offset, HIDDEN, INTER, ws.ptr, ws.nbytes, st["rows_out"].data_ptr(),
        HIDDEN, stream), "b200moe_ep_local_experts")
    out = torch.empty((T, HIDDEN), dtype=torch.bfloat16, device=dev)
    parts = (ctypes.c_void_p * world)(*[p.data_ptr() for p in st["partials"]])
    _capi.check(lib.b200moe_ep_combine_peers(parts, st["starts"].data_ptr(), slot.data_ptr(), T, HIDDEN, world,
                                             out.data_ptr(), stream), "b200moe_ep_combine_peers")
    return {"rows": st["rows_out"], "out": out, "counts": counts, "slot": slot[:T]}


def run(st):
    case = st["case"]
    if case["world"]:
        return _run_rank(st)
    lg, hq, hs = st["tokens"]
    w1, s1, w2, s2 = st["w"]
    if st["out"] is not None:
        return kernel.custom_kernel(lg, st["bias"], hq, hs, w1, s1, w2, s2, case["offset"], RSF, out=st["out"])
    return kernel.run(lg, st["bias"], hq, hs, w1, s1, w2, s2, case["offset"], RSF)


def work(case):
    """Bytes and operations of the layer for the rows and experts that such tokens reach (mean of four seeds)."""
    rows = active = sent = 0.0
    T = case["tokens"] * max(1, case["world"])
    for seed in range(4):
        g = torch.Generator().manual_seed(seed)
        bias = synth.make_bias(seed, case["zipf"])
        ids = _route(_logits(T, bias, case, g, "cpu"), bias)
        here = _local(ids, case)
        rows += here.sum().item() / 4
        active += ids[here].unique().numel() / 4
        if case["world"]:
            own = ids[:case["tokens"]] // case["experts"]
            sent += sum((own == d).any(1).sum().item() for d in range(case["world"])) / 4
            got = here.any(1).sum().item()
    flops = synth.algorithmic_flops(int(rows))
    if not case["world"]:
        nbytes = synth.algorithmic_bytes(case["tokens"], 0) + active * synth.algorithmic_bytes(0, 1)
        return {"bytes": int(nbytes), "flops": flops}
    rb = ep.send_row_bytes(HIDDEN)
    nbytes = case["tokens"] * (HIDDEN + 224 + 1024) + sent * rb          # route and pack
    nbytes += got * (rb + 2 * HIDDEN) + active * synth.algorithmic_bytes(0, 1)   # rows in, partial rows out, weights
    nbytes += sent * 2 * HIDDEN + case["tokens"] * 2 * HIDDEN            # combine
    return {"bytes": int(nbytes), "flops": flops}


def tolerance(case):
    # Against the same layer evaluated in fp64 (e4m3 requantisation kept), these cases measure rel 4.5e-3 ... 7.2e-3 and
    # max up to 0.12: the fp16 activations between the GEMMs, e4m3 codes that flip where sums differ, the bf16 sums.
    return {"rel": 1.5e-2, "max": 0.4}
