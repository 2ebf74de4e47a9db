"""gpt-oss attention of many query rows on the tensor cores (gpt_oss_prefill.cu) against a float64
restatement of RunGptOssAttention (plugins/gpt_oss/cuda/gpt_oss_kernels.cu:125-160,1012-1210), at the
sizes where its tiles can go wrong."""
import math

import pytest
import torch

from garnet_b200 import gpt_oss as go

pytestmark = pytest.mark.gpu
D = torch.float64


def bf(t):
    return t.to(torch.bfloat16).float()


def make(tokens, starts, window, q_heads=64, kv_heads=8, page=16, prefill=1, seed=0, exact=True, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    batch = len(starts)
    logical = (max(starts) + tokens + page - 1) // page + 1
    physical = batch * logical
    table = torch.randperm(physical, generator=torch.Generator().manual_seed(seed)).reshape(batch, logical).to(torch.int32).cuda()
    keys, values = (torch.randn(2, physical, page, kv_heads, 64, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    qkv = torch.randn(batch * tokens, (q_heads + 2 * kv_heads) * 64, device="cuda", generator=g) * scale
    qkv = bf(qkv) if exact else qkv
    starts_t = torch.tensor(starts, dtype=torch.int32, device="cuda")
    return dict(opt=go.options(q_heads=q_heads, kv_heads=kv_heads, layer=1, page_size=page, window=window, prefill=prefill), qkv=qkv,
                keys=keys, values=values, table=table, lengths=starts_t + tokens, starts=starts_t,
                active=torch.ones(batch, dtype=torch.int32, device="cuda"), sinks=torch.randn(q_heads, device="cuda", generator=g),
                batch=batch, tokens=tokens, physical=physical)


def run(c):
    return go.attention(c["opt"], c["qkv"], c["keys"], c["values"], c["table"], c["lengths"], c["starts"], c["active"], c["sinks"],
                        c["batch"], c["tokens"], c["physical"])


def want(c):
    """The rows in float64, from the caches after the append; also the largest |v| of the cache."""
    o = c["opt"]
    q = c["qkv"][:, :o.q_heads * 64].to(D).reshape(c["batch"], c["tokens"], o.q_heads, 64)
    keys, values = c["keys"][1].reshape(-1, o.kv_heads, 64).to(D), c["values"][1].reshape(-1, o.kv_heads, 64).to(D)
    out = torch.zeros(c["batch"], c["tokens"], o.q_heads, 64, dtype=D, device="cuda")
    limit = c["table"].shape[1] * o.page_size
    for b in range(c["batch"]):
        if not int(c["active"][b]):
            continue
        pages = c["table"][b].repeat_interleave(o.page_size).long()
        there = (pages >= 0) & (pages < c["physical"])
        slots = torch.where(there, pages, 0) * o.page_size + torch.arange(limit, device="cuda") % o.page_size
        pos = torch.arange(limit, device="cuda")[None]
        t = torch.arange(c["tokens"], device="cuda")[:, None]
        end = int(c["starts"][b]) + t + 1 if o.prefill else torch.full_like(t, int(c["lengths"][b]))
        see = (pos < end) & there[None] & (end > 0) & (end <= limit)
        if o.window:
            see &= pos >= end - o.window
        for h in range(o.q_heads):
            kv = h // (o.q_heads // o.kv_heads)
            s = (q[b, :, h] @ keys[slots, kv].T / 8.0).masked_fill(~see, -math.inf)
            sink = c["sinks"][h].to(D)
            m = torch.maximum(s.max(dim=1).values, sink)[:, None]
            p = torch.exp(s - m)
            out[b, :, h] = p @ values[slots, kv] / (p.sum(1, keepdim=True) + torch.exp(sink - m))
    return out.reshape(c["batch"] * c["tokens"], -1), float(values.abs().max())


def check(c):
    k0, v0 = c["keys"].clone(), c["values"].clone()
    got = run(c).to(D)
    w, vmax = want(c)
    # one bf16 step of the result, and the fp32 part: exponents of |s| < 64 to 2^-24 each way, p to 2^-18, sums of p v
    assert bool(((got - w).abs() <= 1.01 * 2.0 ** -7 * w.abs() + 2e-5 * vmax).all()), float((got - w).abs().max())
    assert float((got - w.float().to(torch.bfloat16).to(D)).abs().gt(0).double().mean()) < 0.01    # nearly all round alike
    # the appended rows, bit for bit, and nothing else
    o = c["opt"]
    for cache, first in ((k0, o.q_heads), (v0, o.q_heads + o.kv_heads)):
        rows = c["qkv"].reshape(c["batch"], c["tokens"], -1, 64)[:, :, first:first + o.kv_heads].to(torch.bfloat16)
        for b in range(c["batch"]):
            for t in range(c["tokens"] if int(c["active"][b]) else 0):
                at = int(c["starts"][b]) + t
                page = int(c["table"][b, at // o.page_size]) if at // o.page_size < c["table"].shape[1] else -1
                if 0 <= page < c["physical"]:
                    cache[1, page, at % o.page_size] = rows[b, t]
    assert torch.equal(c["keys"], k0) and torch.equal(c["values"], v0)


@pytest.mark.parametrize("tokens,starts,window", [
    (1, [0], 0), (1, [127, 128], 0), (15, [0, 3], 0), (16, [112], 0), (17, [111, 5], 0), (32, [96], 0), (33, [95], 128),
    (64, [0], 1), (129, [0], 128), (130, [126, 511], 0), (200, [300], 128), (640, [0], 0), (300, [77, 0], 129)])
def test_tiles_causal_and_window(tokens, starts, window):
    check(make(tokens, starts, window))


@pytest.mark.parametrize("q_heads,kv_heads,page", [(8, 8, 16), (8, 4, 5), (6, 2, 16), (16, 1, 1), (128, 1, 16), (24, 8, 32)])
def test_head_groups_and_page_sizes(q_heads, kv_heads, page):
    check(make(45, [100, 7], 0, q_heads, kv_heads, page))


def test_two_tiles_per_block():
    """Enough rows that a block takes two tiles of queries, large scores (the running maximum grows), sinks that dominate."""
    c = make(700, [0], 0, scale=3.0, seed=2)
    c["sinks"][::3] = 30.0
    c["sinks"][1::3] = -math.inf
    check(c)


def test_inactive_sequences_missing_pages_and_rows_beyond_the_table():
    c = make(40, [90, 10, 30, 0], 0, seed=3)
    c["active"][1] = 0
    c["table"][2, 1] = -1
    c["table"][0, 4] = c["physical"]
    c["table"] = c["table"][:, :7].contiguous()       # sequence 0 ends past the last logical page
    check(c)


def test_rows_that_see_the_whole_sequence():
    """Several new rows without the causal rule: every row sees `lengths` positions."""
    check(make(5, [123, 0], 0, prefill=0))
    check(make(5, [223, 4], 128, prefill=0))


def test_queries_that_are_not_bf16_values():
    check(make(20, [50], 0, exact=False, seed=4))


def test_infinite_values_stay_infinite():
    c = make(40, [300], 0, seed=5)
    slot = c["table"][0, 3]
    c["values"][1, slot, 2, 0, 7] = math.inf
    c["values"][1, slot, 5, 1, 9] = -math.inf
    got, (w, _) = run(c).to(D).reshape(40, 64, 64), want(c)
    w = w.reshape(40, 64, 64)
    assert bool((got[:, :8, 7] == math.inf).all()) and bool((got[:, 8:16, 9] == -math.inf).all())
    rest = torch.isfinite(w)
    assert torch.equal(torch.isfinite(got), rest) and float((got - w)[rest].abs().max()) < 2e-2


def test_probabilities_keep_their_24_bits():
    """Each row sees two keys whose scores differ by d, with values 1 and -1: the result is tanh(d / 2), the difference of two
    nearly equal probabilities, which shows what of them is left out.  Scores are single exact products; an exponential is good
    to 2^-22 and the result is rounded to bf16 once."""
    c = make(200, [0], 2, seed=7)
    g = torch.Generator().manual_seed(7)
    qkv = torch.zeros(200, 80, 64)
    qkv[:, :64, 3] = bf(1 + torch.rand(200, 64, generator=g))
    qkv[:, 64:72, 3] = 0.125 + torch.randint(0, 32, (200, 8), generator=g) * 2.0 ** -10
    qkv[:, 72:, :] = (1 - 2.0 * (torch.arange(200) % 2)).reshape(-1, 1, 1)
    c["qkv"] = qkv.reshape(200, -1).cuda()
    c["sinks"][:] = -math.inf
    got = run(c).to(D)
    w, _ = want(c)
    assert bool(((got - w).abs() <= 1.01 * 2.0 ** -8 * w.abs() + 2.0 ** -22).all()), float((got - w).abs().max())


def test_an_infinite_sink_gives_what_the_row_loop_gives():
    """exp(inf - inf) is NaN for the heads with the infinite sink; the others are not touched by it."""
    c = make(40, [100], 0, seed=6)
    c["sinks"][5] = math.inf
    got, (w, vmax) = run(c).to(D).reshape(40, 64, 64), want(c)
    w = w.reshape(40, 64, 64)
    assert bool(got[:, 5].isnan().all())
    rest = torch.arange(64, device="cuda") != 5
    assert bool(((got - w)[:, rest].abs() <= 1.01 * 2.0 ** -7 * w[:, rest].abs() + 2e-5 * vmax).all())


def device_us(c, calls=5):
    ws = torch.zeros(1 << 24, dtype=torch.uint8, device="cuda")
    def one():
        go.attention(c["opt"], c["qkv"], c["keys"], c["values"], c["table"], c["lengths"], c["starts"], c["active"], c["sinks"],
                     c["batch"], c["tokens"], c["physical"], workspace=ws)
    one()
    best = math.inf
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(calls):
            one()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 1000 / calls)
    return best


def test_queries_that_are_not_bf16_values_stay_on_the_tensor_cores():
    """Three pieces of each query: two tiles per block, one query alone that needs them, and no row loop over the keys (which
    took some hundred times as long)."""
    check(make(700, [0], 0, exact=False, seed=8))
    c = make(300, [40], 128, seed=9)
    c["qkv"][123, 17 * 64 + 5] += 2.0 ** -12
    check(c)
    plain, pieces = make(512, [0], 0, seed=10), make(512, [0], 0, exact=False, seed=10)
    assert device_us(pieces) < 4 * device_us(plain)


def test_blocks_whose_second_tile_has_no_rows():
    """Sequences of 33 tokens (two blocks of two tiles, the last with one token) and of 16 (one tile), enough to fill the GPU."""
    check(make(33, list(range(0, 200, 10)), 0, seed=11))
    check(make(16, list(range(0, 200, 10)), 0, seed=12))
