"""gpt-oss decode attention (gpt_oss_decode.cu) against a float64 restatement of RunGptOssAttention
(plugins/gpt_oss/cuda/gpt_oss_kernels.cu:125-160,376-535), at the sizes where its tiles of 16 positions, rounds of
warps and clusters can go wrong, and RoPE's two access widths against each other."""
import ctypes
import math

import pytest
import torch

from garnet_b200 import gpt_oss as go
from garnet_b200._lib import check as check_code, lib
from test_gpt_oss_prefill_gpu import D, check, device_us, make, run, want

pytestmark = pytest.mark.gpu


def decode(starts, window=0, **kw):
    return make(1, starts, window, prefill=0, **kw)


@pytest.mark.parametrize("starts,window", [
    ([0], 0), ([14, 15, 16], 0), ([126, 127, 128], 0), ([254, 255, 256, 511, 512, 1023], 0), ([3071, 3072, 383], 0),
    ([8190, 0], 0), ([0, 1, 500], 1), ([126, 127, 128, 2000], 128), ([300, 5], 129), (list(range(100, 500, 17)), 0),
    (list(range(100, 500, 17)) * 6, 200)])
def test_lengths_and_windows(starts, window):
    check(decode(starts, window))


@pytest.mark.parametrize("q_heads,kv_heads,page", [(8, 8, 16), (8, 4, 5), (6, 2, 16), (16, 1, 1), (48, 4, 32), (34, 2, 16)])
def test_head_groups_and_page_sizes(q_heads, kv_heads, page):
    check(decode([200, 7, 1500], 0, q_heads=q_heads, kv_heads=kv_heads, page=page))


def test_sinks_large_scores_and_queries_that_are_not_bf16_values():
    c = decode([700, 63], 0, scale=3.0, seed=2)
    c["sinks"][::3] = 30.0
    c["sinks"][1::3] = -math.inf
    check(c)
    check(decode([700, 63], 0, exact=False, seed=4))


def test_inactive_sequences_missing_pages_and_positions_beyond_the_table():
    c = decode([90, 10, 130, 0, 60], 0, seed=3)
    c["active"][1] = 0
    c["table"][0, 1] = -1
    c["table"][0, 4] = c["physical"]
    c["table"][4, :] = -1                              # nothing but the sink
    c["table"] = c["table"][:, :7].contiguous()        # sequence 2 ends past the last logical page
    check(c)


def test_infinite_values_stay_infinite():
    c = decode([300, 40], 0, seed=5)
    slot = c["table"][0, 3]
    c["values"][1, slot, 2, 0, 7] = math.inf
    c["values"][1, slot, 5, 1, 9] = -math.inf
    got, (w, _) = run(c).to(D).reshape(2, 64, 64), want(c)
    w = w.reshape(2, 64, 64)
    assert bool((got[0, :8, 7] == math.inf).all()) and bool((got[0, 8:16, 9] == -math.inf).all())
    rest = torch.isfinite(w)
    assert torch.equal(torch.isfinite(got), rest) and float((got - w)[rest].abs().max()) < 2e-2


@pytest.mark.parametrize("shift", [1, 2, 3])
def test_operands_aligned_to_their_values_only(shift):
    """Queries and output at any multiple of four bytes, on the same kernel (the row loop takes some fifty times as long)."""
    c = decode([100, 33, 3000], 0, seed=6)
    moved = torch.empty(c["qkv"].numel() + 4, device="cuda")[shift:][:c["qkv"].numel()].view_as(c["qkv"]).copy_(c["qkv"])
    check(dict(c, qkv=moved))
    want_y = run(c)
    y = torch.zeros(want_y.numel() + 8, device="cuda")
    need = ctypes.c_size_t(0)
    logical = c["table"].shape[1]
    check_code(lib().garnet_b200_gpt_oss_attention_workspace(ctypes.byref(c["opt"]), c["batch"], logical, ctypes.byref(need)))
    ws = torch.zeros(need.value, dtype=torch.uint8, device="cuda")
    operands = (ctypes.c_void_p * 8)(*[t.data_ptr() for t in (moved, c["keys"], c["values"], c["table"], c["lengths"], c["starts"],
                                                              c["active"], c["sinks"])])
    check_code(lib().garnet_b200_gpt_oss_attention(ctypes.byref(c["opt"]), operands, y.data_ptr() + 4 * shift, ws.data_ptr(), ws.numel(),
                                                   c["batch"], 1, logical, c["physical"], torch.cuda.current_stream().cuda_stream))
    assert torch.equal(y[shift:shift + want_y.numel()].view_as(want_y), want_y)
    assert not bool(y[:shift].any()) and not bool(y[shift + want_y.numel():].any())
    assert device_us(dict(c, qkv=moved)) < 4 * device_us(c)


def test_rope_access_widths_agree():
    opt = go.options(q_heads=6, kv_heads=2, head_dim=64)
    for tokens in (1, 2, 3, 77, 301):
        x = torch.randn(tokens, 10 * 64, device="cuda").to(torch.bfloat16).float()
        positions = torch.randint(0, 9000, (tokens,), device="cuda")
        moved = torch.empty(x.numel() + 1, device="cuda")[1:].view_as(x).copy_(x)
        assert torch.equal(go.rope(opt, x, positions), go.rope(opt, moved, positions))


@pytest.mark.parametrize("starts,exact,share", [([8190 - i for i in range(16)], True, 4e-4), ([2999, 2500, 2300, 2700] * 4, False, 4.7e-4)])
def test_long_sums_round_as_fp32_sums_do(starts, exact, share):
    """The share of results that are not the bf16 rounding of the float64 result.  Scalar fp32 sums over splits of 64 positions
    leave 2.9e-4 and 4.2e-4 here (of 393216 results, so give or take 4e-5); accumulators that truncate 6.4e-4 and 5.4e-4."""
    wrong = []
    for seed in range(6):
        c = decode(starts, 0, exact=exact, seed=seed)
        got, (w, _) = run(c).to(D), want(c)
        wrong.append(float((got - w.float().to(torch.bfloat16).to(D)).abs().gt(0).double().mean()))
    assert sum(wrong) / len(wrong) < share, wrong
