"""The attention kernel of four chains (d_h 16, 32, 64): against float64 where chains run out of keys at different times, or have none."""
import os
import re

import pytest

from conftest import ROOT


def attention(pkg, torch, q, k, v, q_start, q_rows, split, causal, counters=None):
    H, S, d_h = q.shape
    fp = pkg.FlashParams(S, d_h, H, split, causal, d_h ** -0.5)
    out = torch.full((q_rows, H * d_h), float("nan"), device="cuda")
    ws = [torch.full((n,), float("nan"), device="cuda") for n in (split * q_rows * H * d_h, split * q_rows * H, split * q_rows * H)]
    part = pkg.FlashPartials(*(w.data_ptr() for w in ws), q_rows) if split > 1 else None
    pkg.kernel_status_reset()
    pkg.flash_attn_tc_forward(q, k, v, out, part, q_start, q_rows, fp, tile_counters=counters, tile_rows=64 if counters is not None else 0, o_dtype=pkg.F32)
    if part is not None:
        pkg.flash_attn_tc_combine(part, out, 0, q_rows, fp, o_dtype=pkg.F32)
    torch.cuda.synchronize()
    assert pkg.kernel_status()[0] == 0
    return out, pkg.flash_attn_tc_plan(fp, q_start, q_rows)


def check(torch, out, q, k, v, q_start, q_rows, causal):
    H, S, d_h = q.shape
    rows = torch.arange(q_start, q_start + q_rows, device="cuda")[:, None]
    for h in range(H):
        s = q[h, q_start:q_start + q_rows].double() @ k[h].double().T * d_h ** -0.5
        if causal:
            s = s.masked_fill(torch.arange(S, device="cuda")[None, :] > rows, float("-inf"))
        w = torch.softmax(s, dim=-1)
        ref = w @ v[h].double()
        # every weight is rounded to fp16 (2^-11 of it) or, below 2^-14 of the largest, to a multiple of 2^-25 (the offset may lag the
        # maximum by 2^8); fp32 scores of up to about 100 carry 1e-5 of relative error into the weights
        bound = (w * 2 ** -11 + 2.0 ** -24) @ v[h].double().abs() + 1e-4 * ref.abs().max()
        err = (out[:, h * d_h:(h + 1) * d_h].double() - ref).abs()
        assert bool((err <= bound).all()), (h, float((err - bound).max()))


def launched(plan):
    return "+".join(n for n, items in (("256", plan.items_256), ("128", plan.items_128), ("tiles", plan.tiles)) if items)


@pytest.mark.gpu
# One to nine blocks of 64 keys (chains without a block, ragged halves of a stage), one to four 64-row blocks, and beyond the K/V ring. Two heads: 128-row
# items on four chains. 300: 256-row items on two chains per tile; at d_h 16 and 32, but for the longest, the kernel of one tile.
@pytest.mark.parametrize("d_h", [16, 32, 64])
@pytest.mark.parametrize("H", [2, 300])
@pytest.mark.parametrize("S,q_start,q_rows,split,causal", [(64, 0, 64, 1, 0), (128, 64, 64, 1, 1), (192, 0, 192, 1, 0), (320, 64, 256, 1, 1), (576, 0, 64, 1, 0),
                                                           (1344, 1088, 256, 1, 1), (1152, 1024, 128, 2, 0), (1152, 512, 192, 3, 1)])
def test_blocks_of_keys_and_rows(pkg, torch_cuda, d_h, H, S, q_start, q_rows, split, causal):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(S + d_h)
    q, k, v = (torch.randn(H, S, d_h, generator=g, device="cuda", dtype=torch.float16) for _ in range(3))
    counters = torch.zeros(q_rows // 64, dtype=torch.int32, device="cuda")
    out, plan = attention(pkg, torch, q, k, v, q_start, q_rows, split, causal, counters)
    assert launched(plan) == ("128" if H == 2 else "256" if d_h == 64 or S == 1344 else "tiles")
    check(torch, out, q, k, v, q_start, q_rows, causal)
    assert counters.tolist() == [H * split] * (q_rows // 64)


@pytest.mark.gpu
# Two chains per tile with as few keys, at all head sizes: chains without a block (320), 64 rows in the second tile, a split that has keys for 64 of 256 rows, ragged splits.
@pytest.mark.parametrize("d_h", [16, 32, 64])
@pytest.mark.parametrize("S,q_start,q_rows,split,causal", [(320, 64, 256, 1, 1), (448, 256, 192, 1, 0), (640, 320, 192, 1, 0), (1024, 320, 256, 2, 1),
                                                           (1152, 640, 192, 2, 1)])
def test_two_chains_per_tile_with_few_keys(pkg, torch_cuda, d_h, S, q_start, q_rows, split, causal):
    torch = torch_cuda
    H = 140 // split
    g = torch.Generator(device="cuda").manual_seed(S + d_h)
    q, k, v = (torch.randn(H, S, d_h, generator=g, device="cuda", dtype=torch.float16) for _ in range(3))
    for counters in (None, torch.zeros(q_rows // 64, dtype=torch.int32, device="cuda")):
        out, plan = attention(pkg, torch, q, k, v, q_start, q_rows, split, causal, counters)
        assert launched(plan) == "256"
        check(torch, out, q, k, v, q_start, q_rows, causal)
    assert counters.tolist() == [H * split] * (q_rows // 64)


@pytest.mark.gpu
# 128-row items, 256-row items, the kernel of one tile, and splits
@pytest.mark.parametrize("d_h,H,S,split,want", [(16, 2, 512, 1, "128"), (32, 2, 1024, 2, "128"), (64, 2, 512, 1, "128"), (16, 74, 512, 1, "256"), (32, 148, 512, 1, "256"),
                                                (64, 300, 512, 1, "256"), (64, 100, 1024, 2, "256"), (32, 200, 256, 1, "tiles"), (128, 2, 512, 1, "128"), (128, 150, 512, 1, "256")])
@pytest.mark.parametrize("causal", [0, 1])
def test_infinite_scores(pkg, torch_cuda, d_h, H, S, split, want, causal):
    """Keys that score -inf have no weight, whichever chains have nothing else; a row that has a key scoring +inf, or none but such scoring -inf, is no number."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(S + d_h)
    q, k, v = (torch.randn(H, S, d_h, generator=g, device="cuda", dtype=torch.float16) for _ in range(3))
    q[..., 0] = q[..., 0].abs() + 0.125
    block = torch.arange(S, device="cuda") // 64
    assert launched(attention(pkg, torch, q, k, v, 0, S, split, 0)[1]) == want
    for gone in (block == 1, block % 2 == 1, block % 4 != 0, (block % 2 == 0) & (torch.arange(S, device="cuda") > 0), torch.arange(S, device="cuda") >= 3):
        x = k.clone()
        x[:, gone, 0] = float("-inf")
        out, _ = attention(pkg, torch, q, x, v, 0, S, split, causal)
        check(torch, out, q, x, v, 0, S, causal)
    x = k.clone()
    x[:, S // 2 + 70, 0] = float("inf")
    out, _ = attention(pkg, torch, q, x, v, 0, S, split, causal)
    seen = S // 2 + 70 if causal else 0
    assert torch.isnan(out[seen:]).all() and torch.isfinite(out[:seen]).all()
    x[..., 0] = float("-inf")
    out, _ = attention(pkg, torch, q, x, v, 0, S, split, causal)
    assert torch.isnan(out).all()


@pytest.mark.gpu
@pytest.mark.parametrize("d_h,H,items128", [(64, 2, True), (64, 300, False), (16, 2, True), (32, 300, False)])
def test_chains_whose_maxima_lie_far_apart(pkg, torch_cuda, d_h, H, items128):
    """Each chain's keys score on a level of their own, up to 2^60 apart, which level is the highest changing with the row."""
    torch = torch_cuda
    S, rows = 1024, 256
    g = torch.Generator(device="cuda").manual_seed(d_h)
    q, k, v = (torch.randn(H, S, d_h, generator=g, device="cuda", dtype=torch.float16) for _ in range(3))
    level = torch.tensor([0.0, 3.0, -2.0, 1.0], device="cuda").repeat_interleave(64).repeat(S // 256)     # by block of 64 keys
    k[..., 0] = level.half()
    q[..., 0] = (torch.arange(S, device="cuda") % 7 - 3).half() * d_h ** 0.5
    out, plan = attention(pkg, torch, q, k, v, 0, rows, 1, 0)
    assert (plan.items_128 > 0) == items128
    check(torch, out, q, k, v, 0, rows, 0)


def test_the_kernel_presumes_no_read_only_memory():
    """It starts before the kernel ahead of it has ended (launch_early), like the one it shares its name with."""
    with open(os.path.join(ROOT, "eager-flash-attention_b200", "csrc", "fa_fwd_chains.cuh")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    assert not re.search(r"__restrict__|__ldg\b|\.nc\b|__constant__", text)
    assert text.index("pdl_wait()") < text.index("pdl_trigger()") < text.index("tma_load_3d(")
