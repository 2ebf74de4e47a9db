"""The workloads that this library's speed is judged by: what its users have it do, at the sizes they do it.

Five kinds of call, each through the Python face of the C ABI:

  linear     one int4 linear, W4A16Linear.forward: any projection of a Qwen3-1.7B decoder (or a ragged width),
             1 row (decode) up to a prefill chunk of about a thousand rows, bf16 or fp16 group scales
  pass       every int4 linear of a decode step as one prepared list, LinearList.run (197 linears for 28 layers)
  step       a whole greedy decode step, DecodeStep.run: embedding to arg-max, paged KV cache, 1 to 8 sequences
  moe        the gpt-oss-120b mixture-of-experts layer, GptOssMoe.run: 1 token up to a 4096-token prefill,
             fp32 carrier or bf16, evenly popular experts or popularity after Zipf's law
  attention  the gpt-oss-120b attention of one layer, gpt_oss.rope + gpt_oss.attention: decode of a batch of
             ragged sequences, prefill of a prompt or of a further chunk of it, full or with the sliding window
"""
from __future__ import annotations

import math

import numpy as np
import torch

import garnet_b200 as gb
from garnet_b200 import decode, gpt_oss, synth

GROUP = 128
MOE = dict(hidden=2880, inter=2880, experts=128, top_k=4)
OSS_Q, OSS_KV, OSS_DIM, OSS_PAGE, OSS_WINDOW = 64, 8, 64, 16, 128
# (k, n) of the Qwen3-1.7B projections: q and o, k and v, packed q/k/v, gate or up, packed gate/up, down
PROJECTIONS = [(2048, 2048), (2048, 1024), (2048, 4096), (2048, 6144), (2048, 12288), (6144, 2048)]
LM_HEAD = (2048, 151936)


def listed():
    return [
        # one projection of one token: the smallest call there is, launch and host path count
        dict(name="linear gate m1", kind="linear", n=6144, k=2048, m=1, scales="bf16"),
        # a decode batch of 16 sequences on the projection with the long K
        dict(name="linear down m16", kind="linear", n=2048, k=6144, m=16, scales="bf16"),
        # a short prompt: ragged rows on packed q/k/v, scales as the reference's artifacts store them
        dict(name="linear qkv m77", kind="linear", n=4096, k=2048, m=77, scales="fp16"),
        # a prefill chunk on the widest projection of a layer
        dict(name="linear gate_up m1000", kind="linear", n=12288, k=2048, m=1000, scales="bf16"),
        # all linears of one decode token: the headline workload of the benchmark
        dict(name="pass 28 layers m1", kind="pass", layers=28, m=1),
        # one greedy token of one sequence after a context of 2048
        dict(name="step b1 ctx2048", kind="step", batch=1, context=2048),
        # decode of one sequence: the four routed experts are all there is to read
        dict(name="moe t1", kind="moe", tokens=1, io="fp32", routing="even"),
        # a decode batch
        dict(name="moe t32", kind="moe", tokens=32, io="bf16", routing="even"),
        # a short prompt with skewed experts
        dict(name="moe t500 zipf", kind="moe", tokens=500, io="fp32", routing="zipf"),
        # a prefill chunk
        dict(name="moe t4096", kind="moe", tokens=4096, io="bf16", routing="even"),
        # decode attention of four ragged sequences
        dict(name="attention decode b4", kind="attention", phase="decode", batch=4, tokens=1, start=2999, window=0),
        # prefill of one prompt
        dict(name="attention prefill 2048", kind="attention", phase="prefill", batch=1, tokens=2048, start=0, window=0),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "pass", "step", "moe", "moe", "moe", "attention", "attention", "attention"])
    if kind == "linear":
        pick = rng.randrange(8)
        if pick == 6:                       # lm_head: logits of a batch, never of a whole prompt
            k, n, most = *LM_HEAD, 256
        elif pick == 7:                     # a ragged width (a shard of a projection, another model's head count)
            k, n, most = 128 * rng.randint(4, 48), rng.randint(200, 12288), 1024
        else:
            (k, n), most = PROJECTIONS[pick], 1024
        return dict(kind=kind, n=n, k=k, m=_log_int(rng, 1, most), scales=rng.choice(["bf16", "bf16", "fp16"]))
    if kind == "pass":
        return dict(kind=kind, layers=rng.randint(4, 28), m=rng.randint(1, 8))
    if kind == "step":
        return dict(kind=kind, batch=rng.randint(1, 8), context=_log_int(rng, 64, 4096))
    if kind == "moe":
        return dict(kind=kind, tokens=_log_int(rng, 1, 4096), io=rng.choice(["fp32", "bf16"]), routing=rng.choice(["even", "zipf"]))
    window = rng.choice([0, OSS_WINDOW])
    if rng.random() < 0.5:
        return dict(kind=kind, phase="decode", batch=rng.randint(1, 16), tokens=1, start=_log_int(rng, 16, 8191), window=window)
    tokens, batch = _log_int(rng, 32, 2048), rng.randint(1, 4)
    start = rng.choice([0, rng.randint(1, 2048)])
    while batch > 1 and batch * tokens * (start + tokens) > 2048 * 2048:
        batch -= 1
    start = max(0, min(start, 2048 * 2048 // (batch * tokens) - tokens))
    return dict(kind=kind, phase="prefill", batch=batch, tokens=tokens, start=start, window=window)


# ------------------------------------------------------------------ inputs


def _gen(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return gen


def _normal(gen, *shape):
    return torch.randn(*shape, device="cuda", generator=gen).to(torch.bfloat16)


def _linear(gen, n, k, scale_dtype=torch.bfloat16):
    """Codes uniform in -8..7, group scales |N(0, 0.02)| / 7."""
    nibbles = torch.randint(0, 256, (n * k // 2,), dtype=torch.uint8, device="cuda", generator=gen)
    scales = (torch.randn(n, k // GROUP, device="cuda", generator=gen).abs() * (0.02 / 7.0)).to(scale_dtype)
    return gb.W4A16Linear().prepare(nibbles, scales, n, k, GROUP)


def _pages(count, seed):
    """Physical pages in the order a running server would have handed them out: no order."""
    return torch.from_numpy(np.random.RandomState(seed).permutation(count).astype(np.int32)).cuda()


def _prepare_linear(case, gen):
    lin = _linear(gen, case["n"], case["k"], torch.float16 if case["scales"] == "fp16" else torch.bfloat16)
    return dict(lin=lin, x=_normal(gen, case["m"], case["k"]))


def _prepare_pass(case, gen):
    layers, m = case["layers"], case["m"]
    new = lambda *shape: torch.empty(*shape, dtype=torch.bfloat16, device="cuda")   # noqa: E731
    hidden, inter = _normal(gen, m, 2048), _normal(gen, m, 6144)
    outs = {name: new(layers, m, n) for name, _, n in synth.QWEN3_1P7B_PROJECTIONS}
    outs["lm_head"] = new(m, LM_HEAD[1])
    calls = []
    for i in range(layers):
        for name, k, n in synth.QWEN3_1P7B_PROJECTIONS:
            calls.append((_linear(gen, n, k), inter if k == 6144 else hidden, outs[name][i]))
    calls.append((_linear(gen, LM_HEAD[1], LM_HEAD[0]), hidden, outs["lm_head"]))
    return dict(list=gb.LinearList(calls, m=m), outs=outs)


def _contexts(batch, context, seed):
    """Ragged lengths of a batch: the first sequence is the longest."""
    r = np.random.RandomState(seed)
    return [context] + [int(r.randint(max(1, context // 2), context + 1)) for _ in range(batch - 1)]


def _prepare_step(case, gen, seed):
    cfg = decode.DecoderConfig()
    batch, context = case["batch"], case["context"]
    pages = (context + cfg.page_size - 1) // cfg.page_size
    weights = decode.synthetic_decoder(cfg, seed=seed)
    keys, values = (_normal(gen, cfg.layers, batch * pages, cfg.page_size, cfg.kv_heads, cfg.head_dim) for _ in range(2))
    step = decode.DecodeStep(cfg, weights, batch, max_context=context, key_pages=keys, value_pages=values,
                             page_tables=_pages(batch * pages, seed).reshape(batch, pages))
    step.token_in.copy_(torch.randint(0, cfg.vocab, (batch,), device="cuda", generator=gen))
    step.positions.copy_(torch.tensor([c - 1 for c in _contexts(batch, context, seed)], dtype=torch.int32))
    step.capture()
    return dict(step=step, keys=keys, values=values)


def _prepare_moe(case, gen, seed):
    h, i, e = MOE["hidden"], MOE["inter"], MOE["experts"]
    u8 = lambda lo, hi, *shape: torch.randint(lo, hi, shape, dtype=torch.uint8, device="cuda", generator=gen)   # noqa: E731
    router_w = _normal(gen, e, h).float() / math.sqrt(h)
    router_b = torch.from_numpy(_popularity(case["routing"], np.random.RandomState(seed))).cuda()
    io = torch.float32 if case["io"] == "fp32" else torch.bfloat16
    moe = gb.GptOssMoe(h, i, e, MOE["top_k"], io_dtype=io).prepare(
        router_w.to(torch.bfloat16), router_b.to(torch.bfloat16),
        u8(0, 256, e, 2 * i, h // 32, 16), u8(117, 124, e, 2 * i, h // 32), _normal(gen, e, 2 * i) * 0.1,
        u8(0, 256, e, h, i // 32, 16), u8(117, 124, e, h, i // 32), _normal(gen, e, h) * 0.1)
    return dict(moe=moe, x=_normal(gen, case["tokens"], h).to(io))


def _popularity(routing, r):
    """Router bias of each expert: none, or the logarithm of its share under Zipf(1.1)."""
    e = MOE["experts"]
    if routing == "even":
        return np.zeros(e, np.float32)
    share = (r.permutation(e) + 1.0) ** -1.1
    return np.log(share / share.sum() * e).astype(np.float32)


def _prepare_attention(case, gen, seed):
    batch, tokens, start = case["batch"], case["tokens"], case["start"]
    pages = (start + tokens + OSS_PAGE - 1) // OSS_PAGE
    keys, values = (_normal(gen, 1, batch * pages, OSS_PAGE, OSS_KV, OSS_DIM) for _ in range(2))
    if case["phase"] == "decode":
        starts = [c - 1 for c in _contexts(batch, start + 1, seed)]
    else:
        starts = [start] * batch
    positions = (torch.tensor(starts).reshape(-1, 1) + torch.arange(tokens)).reshape(-1).cuda()
    starts = torch.tensor(starts, dtype=torch.int32).cuda()
    opt = gpt_oss.options(q_heads=OSS_Q, kv_heads=OSS_KV, head_dim=OSS_DIM, page_size=OSS_PAGE, window=case["window"],
                          prefill=1 if case["phase"] == "prefill" else 0)
    return dict(opt=opt, qkv=_normal(gen, batch * tokens, (OSS_Q + 2 * OSS_KV) * OSS_DIM).float(), positions=positions,
                keys=keys, values=values, table=_pages(batch * pages, seed).reshape(batch, pages), starts=starts,
                lengths=starts + tokens, active=torch.ones(batch, dtype=torch.int32, device="cuda"),
                sinks=torch.randn(OSS_Q, device="cuda", generator=gen), batch=batch, tokens=tokens, pages=batch * pages,
                workspace=_attention_workspace(opt, batch, pages))


def _attention_workspace(opt, batch, logical_pages):
    import ctypes
    need = ctypes.c_size_t(0)
    gb._lib.check(gb.lib().garnet_b200_gpt_oss_attention_workspace(ctypes.byref(opt), batch, logical_pages, ctypes.byref(need)))
    return torch.zeros(need.value, dtype=torch.uint8, device="cuda")


def prepare(case, seed):
    gen = _gen(seed)
    kind = case["kind"]
    if kind == "linear":
        state = _prepare_linear(case, gen)
    elif kind == "pass":
        state = _prepare_pass(case, gen)
    elif kind == "step":
        state = _prepare_step(case, gen, seed)
    elif kind == "moe":
        state = _prepare_moe(case, gen, seed)
    else:
        state = _prepare_attention(case, gen, seed)
    state["kind"] = kind
    return state


# ------------------------------------------------------------------ one pass


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["lin"].forward(state["x"])
    if kind == "pass":
        state["list"].run()
        return state["outs"]
    if kind == "step":
        state["step"].run()
        # the logits and the caches; the token is the arg-max of the logits, which near-ties make a matter of the last bit
        return dict(logits=state["step"].logits, keys=state["keys"], values=state["values"])
    if kind == "moe":
        return state["moe"].run(state["x"])
    s = state
    rotated = gpt_oss.rope(s["opt"], s["qkv"], s["positions"])
    y = gpt_oss.attention(s["opt"], rotated, s["keys"], s["values"], s["table"], s["lengths"], s["starts"], s["active"], s["sinks"],
                          s["batch"], s["tokens"], s["pages"], workspace=s["workspace"])
    return dict(y=y, keys=s["keys"], values=s["values"])


# ------------------------------------------------------------------ what a pass cannot do without


def _linear_work(n, k, m, activations=True):
    return n * k // 2 + n * (k // GROUP) * 2 + (m * k * 2 + m * n * 2 if activations else 0), 2 * m * n * k


def _moe_work(case):
    """Weights of the experts that are routed to (their number from a simulated routing), rows in and out."""
    h, i, e, t = MOE["hidden"], MOE["inter"], MOE["experts"], case["tokens"]
    r = np.random.RandomState(1)
    logits = r.standard_normal((t, e)) + _popularity(case["routing"], r)
    distinct = len(np.unique(np.argpartition(-logits, MOE["top_k"], axis=1)[:, :MOE["top_k"]]))
    per_expert = (2 * i * h + h * i) // 2 + (2 * i * h + h * i) // 32 + (2 * i + h) * 4
    nbytes = distinct * per_expert + e * h * 4 + t * h * 2 * (4 if case["io"] == "fp32" else 2)
    return nbytes, t * (MOE["top_k"] * 2 * 3 * h * i + 2 * e * h)


def _attention_work(case):
    batch, tokens, start, window = case["batch"], case["tokens"], case["start"], case["window"]
    width = (OSS_Q + 2 * OSS_KV) * OSS_DIM
    if case["phase"] == "decode":
        lengths = [0.75 * (start + 1)] * batch
        lengths[0] = start + 1
        seen = sum(min(c, window) if window else c for c in lengths)      # (query, key) pairs
        read = seen
    else:
        ends = np.arange(start + 1, start + tokens + 1)
        seen = batch * int((np.minimum(ends, window) if window else ends).sum())
        read = batch * (min(start, window) if window else start)           # cached positions; the new ones arrive in qkv
    kv = 2 * OSS_KV * OSS_DIM * 2
    rows = batch * tokens
    return rows * width * 4 + rows * OSS_Q * OSS_DIM * 4 + rows * kv + read * kv, 4 * OSS_Q * OSS_DIM * seen


def work(case):
    kind = case["kind"]
    if kind == "linear":
        nbytes, flops = _linear_work(case["n"], case["k"], case["m"])
    elif kind in ("pass", "step"):
        cfg, m = decode.DecoderConfig(), case["m"] if kind == "pass" else case["batch"]
        layers = case["layers"] if kind == "pass" else cfg.layers
        nbytes, flops = _linear_work(LM_HEAD[1], LM_HEAD[0], m)
        for _, k, n in synth.QWEN3_1P7B_PROJECTIONS:
            b, f = _linear_work(n, k, m, activations=kind == "pass")
            nbytes, flops = nbytes + layers * b, flops + layers * f
        if kind == "step":
            seen = case["context"] * (1 + 0.75 * (m - 1))
            nbytes += layers * seen * cfg.kv_heads * cfg.head_dim * 2 * 2
            flops += layers * seen * cfg.q_heads * cfg.head_dim * 4
    elif kind == "moe":
        nbytes, flops = _moe_work(case)
    else:
        nbytes, flops = _attention_work(case)
    return {"bytes": int(nbytes), "flops": int(flops)}


def tolerance(case):
    """About four times what the path differs by from a float64 restatement with the same bf16 rounding points."""
    kind = case["kind"]
    if kind in ("linear", "pass"):
        # bf16 results; above 16 rows also weights rounded once to bf16 (seen: 2.6e-3, worst value 1.3e-2)
        return {"rel": 8e-3, "max": 3e-2}
    if kind == "step":
        # 28 layers, each of which rounds its results to bf16 (seen: 1.3e-2, worst value 7e-2)
        return {"rel": 3e-2, "max": 3e-1}
    if kind == "moe":
        # bf16 roundings of the hidden rows, the experts' values and their sum (seen: 5e-3, worst value 3.1e-2)
        return {"rel": 1e-2, "max": 1e-1}
    # fp32 sums, of which one in some hundreds rounds to the other bf16 neighbour (seen: 5e-5, worst value 7.8e-3)
    return {"rel": 4e-4, "max": 3e-2}
